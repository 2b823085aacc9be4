"""lc_broadphase_update_host with page-locked arrays: they are the caller's again
when the call returns, also while the stream still has earlier work to do."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from licenta_gb300 import _ffi
from licenta_gb300.broadphase import Broadphase
from oracle.broadphase import box_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["brute", "sap", "grid", "hash", "bvh"])
def test_arrays_may_be_reused_after_the_update(cuda, method):
    torch = cuda
    n = 3000
    rng = np.random.default_rng(4)
    lo = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    hi = lo + np.float32(0.04)
    want = box_pairs(lo, hi)
    assert len(want) > 100
    plo, phi = (torch.from_numpy(a.copy()).pin_memory() for a in (lo, hi))
    stream = torch.cuda.Stream()
    bp = Broadphase(method, n, cells_per_axis=24, cell_size=0.04, table_size=1 << 14, max_entries=1 << 20)
    L, got = _ffi.lib(), C.c_uint64()
    st = C.c_void_p(stream.cuda_stream)
    out = np.zeros((2 * len(want), 2), np.uint32)
    try:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # some 10 ms of earlier work
        _ffi.check(L.lc_broadphase_update_host(bp._h, C.c_void_p(plo.data_ptr()), C.c_void_p(phi.data_ptr()), n, st),
                   "update_host")
        plo.copy_(torch.arange(3 * n, dtype=torch.float32).reshape(n, 3))  # the next frame: far apart
        phi.copy_(plo)
        _ffi.check(L.lc_broadphase_test_host(bp._h, out.ctypes.data_as(C.c_void_p), len(out), C.byref(got), st),
                   "test_host")
    finally:
        bp.close()
    p = out[: got.value]
    assert np.array_equal(p[np.lexsort((p[:, 1], p[:, 0]))], want)
