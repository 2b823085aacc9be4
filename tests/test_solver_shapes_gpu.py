"""The on-chip solver's launch shapes: cluster sizes on cloths smaller than a
cluster, and the block size a batch picks from how many cloths it holds.  The
scatter solver sums fixed-point corrections, so its bits do not depend on the
shape; against the global-memory solver (float sums in another order) the
bound is that of the parity tests, 1e-5 m."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, _ffi, scenes

pytestmark = pytest.mark.gpu


def _cluster_size(batch: ClothBatch, cs: int) -> None:
    t = _ffi.Tuning()
    _ffi.check(_ffi.lib().lc_batch_get_tuning(batch._h, C.byref(t)), "lc_batch_get_tuning")
    t.cluster_size = cs
    _ffi.check(_ffi.lib().lc_batch_set_tuning(batch._h, C.byref(t)), "lc_batch_set_tuning")


def _step(specs, steps: int, cs: int = 0, **kw):
    with ClothBatch(specs, **kw) as b:
        if cs:
            _cluster_size(b, cs)
        b.step(steps)
        b.sync()
        return [b.get_state(c) for c in range(len(specs))]


def _triangle():
    s = scenes.small_cloth(seed=3, n=2)
    return scenes.ClothSpec(s.positions[:3], s.indices[:1] * 0 + np.arange(3, dtype=np.uint32), s.pinned[:3], s.params)


@pytest.mark.parametrize("side", [1, 2, 3, 4, 5, 7])
def test_cloths_smaller_than_a_cluster(cuda, side):
    spec = _triangle() if side == 1 else scenes.small_cloth(seed=side, n=side)
    want = _step([spec], 2, solver_variant=1)[0]
    first = None
    for cs in (4, 8, 16):
        got = _step([spec], 2, cs=cs, solver_variant=3)[0]
        assert np.abs(got["x"] - want["x"]).max() < 1e-5
        first = got if first is None else first
        for k in ("x", "x_prev", "v"):
            assert np.array_equal(got[k].view(np.uint32), first[k].view(np.uint32)), (cs, k)


@pytest.mark.parametrize("side,copies", [(24, 96), (64, 40), (101, 24)])
def test_a_cloth_alone_equals_the_cloth_in_a_full_batch(cuda, side, copies):
    """Alone it takes large blocks, in a batch that fills the chip small ones."""
    spec = scenes.small_cloth(seed=side, n=side, thickness=0.3 / side)
    alone = _step([spec], 3)[0]
    for st in (q := _step([spec] * copies, 3))[:: max(1, len(q) // 4)]:
        for k in ("x", "x_prev", "v"):
            assert np.array_equal(st[k].view(np.uint32), alone[k].view(np.uint32)), k
