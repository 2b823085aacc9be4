"""Object broadphase over sizes around a warp, a block and a sort tile, with
boxes that only touch: device and host entries give the brute-force pairs."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from licenta_gb300 import _ffi
from licenta_gb300.broadphase import Broadphase
from oracle.broadphase import box_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["brute", "sap", "grid", "hash", "bvh"])
@pytest.mark.parametrize("n", [2, 3, 31, 33, 257, 2049, 4097])
def test_sizes(method, n):
    rng = np.random.default_rng(n)
    side = max(2, round(n ** (1 / 3)))
    lo = (rng.integers(0, side, (n, 3)) / np.float32(side)).astype(np.float32)  # many faces in common
    hi = lo + np.float32(1 / side)
    want = box_pairs(lo, hi)
    bp = Broadphase(method, n, cells_per_axis=24, cell_size=0.04, table_size=1 << 14, max_entries=1 << 22)
    try:
        bp.update(torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda())
        dev = bp.test().cpu().numpy()
        tests = bp.criteria()["intersection_tests"]
        L, n_out = _ffi.lib(), C.c_uint64()
        ptr = lambda a: a.ctypes.data_as(C.c_void_p)
        _ffi.check(L.lc_broadphase_update_host(bp._h, ptr(lo), ptr(hi), n, None), "update_host")
        host = np.full((len(dev) + 1, 2), 0xFFFFFFFF, np.uint32)
        _ffi.check(L.lc_broadphase_test_host(bp._h, ptr(host), len(host), C.byref(n_out), None), "test_host")
        assert n_out.value == len(dev)
        assert bp.criteria()["intersection_tests"] == tests
    finally:
        bp.close()
    assert np.array_equal(dev, host[:len(dev)])
    p = dev[np.lexsort((dev[:, 1], dev[:, 0]))] if len(dev) else dev.reshape(0, 2)
    assert np.array_equal(p, want)
    if method == "brute":
        assert tests == n * (n - 1) // 2
