"""Creating a batch of the global-memory solver does not pay for tiles that a
vertex of many constraints rules out."""
from __future__ import annotations

import time

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, scenes

pytestmark = pytest.mark.gpu


def _fan(spokes: int):
    a = np.arange(spokes) * (2 * np.pi / spokes)
    rim = np.stack([0.7 + 0.4 * np.cos(a), 1.5 + 0.02 * np.sin(3 * a), 0.7 + 0.4 * np.sin(a)], 1)
    k = np.arange(spokes, dtype=np.uint32)
    tri = np.stack([np.zeros(spokes, np.uint32), 1 + k, 1 + (k + 1) % spokes], 1)
    base = scenes.small_cloth(n=4, iterations=4, stiffness=0.3, thickness=1e-5)
    return scenes.ClothSpec(np.concatenate([[[0.7, 1.5, 0.7]], rim]).astype(np.float32), tri,
                            np.zeros(spokes + 1, base.pinned.dtype), base.params)


def test_a_hub_beside_a_large_cloth(cuda):
    """Six times the time when every size of tile was tried; the bound is 2."""
    big = scenes.large_cloth(seed=1, n=400)
    best = []
    for specs in ([big], [big, _fan(600)]):
        times = []
        for _ in range(4):
            t = time.perf_counter()
            ClothBatch(specs, solver_variant=1).close()
            times.append(time.perf_counter() - t)
        best.append(min(times))
    assert best[1] < 2 * best[0], best
