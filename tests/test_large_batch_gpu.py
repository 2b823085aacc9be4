"""Batches of more than a million leaves: every cloth's pairs and state are the
bits of the same cloth alone, also where the pair chunk of a triangle is
full."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [64, 10])
@pytest.mark.parametrize("side,copies", [(191, 15), (190, 15), (64, 133)])
def test_a_cloth_in_a_large_batch_equals_the_cloth_alone(cuda, side, copies, chunk):
    spec = scenes.small_cloth(seed=side, n=side, thickness=0.6 / side)
    spec.params.BVHChunkSize = chunk
    assert copies * spec.indices.size // 3 > 1 << 20
    out = []
    for n in (1, copies):
        with ClothBatch([spec] * n) as b:
            b.step(2)
            b.sync()
            out.append(([b.get_state(c) for c in range(n)], b.counters()))
    (alone,), one = out[0]
    for st in out[1][0]:
        for k in ("x", "x_prev", "v"):
            assert np.array_equal(st[k].view(np.uint32), alone[k].view(np.uint32)), k
    for k in ("pairs", "vf", "ee", "dropped"):
        assert out[1][1][k] == copies * one[k], k
    assert (one["dropped"] > 0) == (chunk == 10)
