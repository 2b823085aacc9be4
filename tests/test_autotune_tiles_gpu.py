"""The autotuner times the global-memory solver once, not per Jacobi block,
where it works in tiles, and per block where it does not."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, autotune, scenes

pytestmark = pytest.mark.gpu

SPACE = {"traverse_block": (64, 128), "jacobi_block": (128, 256, 512), "narrow_blocks_per_sm": (8,), "solver_variant": (1,)}


def _fan(spokes: int):
    a = np.arange(spokes) * (2 * np.pi / spokes)
    rim = np.stack([0.7 + 0.4 * np.cos(a), 1.5 + 0.02 * np.sin(3 * a), 0.7 + 0.4 * np.sin(a)], 1)
    k = np.arange(spokes, dtype=np.uint32)
    tri = np.stack([np.zeros(spokes, np.uint32), 1 + k, 1 + (k + 1) % spokes], 1)
    base = scenes.small_cloth(n=4, iterations=4, stiffness=0.3, thickness=1e-5)
    return scenes.ClothSpec(np.concatenate([[[0.7, 1.5, 0.7]], rim]).astype(np.float32), tri,
                            np.zeros(spokes + 1, base.pinned.dtype), base.params)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("tiled", [True, False])
def test_trials(cuda, variant, tiled):
    spec = scenes.small_cloth(seed=3, n=24) if tiled else _fan(600)
    with ClothBatch([spec], solver_variant=variant) as b:
        r = autotune.autotune(b, steps=1, warmup=1, space=SPACE, cache=None)
    blocks = [t["config"]["jacobi_block"] for t in r["tried"]]
    assert blocks == ([128] * 2 if tiled else [128, 256, 512] * 2)
