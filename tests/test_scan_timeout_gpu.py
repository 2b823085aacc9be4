"""A scan's wait that gives up is reported by the entries that read their
results back.  The scan itself is a stand-in that sets the error bit
(tests/cpp/scan_gives_up.cu); the entries are the engine's objects."""
from __future__ import annotations

import ctypes as C
import subprocess

import pytest

from licenta_gb300 import _build, _ffi

pytestmark = pytest.mark.gpu

TIMEOUT = 4  # LC_ERR_TIMEOUT


@pytest.fixture(scope="module")
def entries(tmp_path_factory):
    d = tmp_path_factory.mktemp("scan")
    so = d / "libscan_gives_up.so"
    flags = [_build.nvcc(), _build.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I",
             str(_build.REPO / "include")]
    objs = [str(_build.OUT / f"{k}.o") for k in ("lc_response", "lc_static", "lc_lbvh")]
    src = _build.REPO / "tests" / "cpp" / "scan_gives_up.cu"
    r = subprocess.run(flags + ["-shared", "-Xlinker", "-Bsymbolic", "-cudart", "shared", "-o", str(so), str(src)] + objs,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(so))


def _vp(t):
    return C.c_void_p(t.data_ptr())


def test_allocation_free_lbvh(cuda, entries):
    torch = cuda
    n = 700
    lo = torch.rand((n, 3), generator=torch.Generator().manual_seed(1)).cuda()
    hi = lo + 0.05
    pairs, count = torch.zeros((64 * n, 2), dtype=torch.int32, device="cuda"), C.c_uint64()

    def call():
        return entries.lc_lbvh_pairs_static(_vp(lo), _vp(hi), n, 64, _ffi.LC_MORTON_REF63, _vp(pairs), C.c_uint64(64 * n),
                                            C.byref(count), None, None)

    entries.set_give_up(0)
    assert call() == 0 and count.value > 0
    entries.set_give_up(1)
    assert call() == TIMEOUT
    entries.set_give_up(0)
    assert call() == 0
