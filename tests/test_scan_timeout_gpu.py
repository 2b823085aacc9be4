"""A scan's wait that gives up is reported by the entries that read their
results back.  The scan itself is a stand-in that sets the error bit
(tests/cpp/scan_gives_up.cu); the entries are the engine's objects."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from licenta_gb300 import _build, _ffi

pytestmark = pytest.mark.gpu

TIMEOUT, INVALID = 4, 1  # LC_ERR_TIMEOUT, LC_ERR_INVALID_ARG


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


def test_impulse_response(cuda, entries):
    torch = cuda
    V, contacts = 400, 900
    rng = np.random.default_rng(3)
    x = rng.uniform(0, 1, (V, 3)).astype(np.float32)
    rec = np.zeros((contacts, 12), np.int32)
    rec[:, :4] = np.stack([rng.permutation(V)[:4] for _ in range(contacts)])
    f = rec.view(np.float32)
    f[:, 4:8] = 0.25
    f[:, 9] = 1.0
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dx, dxp, fixed = dev(x), dev(x - np.float32(0.001)), dev(np.zeros(V, np.uint8))
    prm = [C.c_float(k) for k in (0.9, 0.01, 1 / 60, 0.02)]

    def call(records):
        r, v = dev(records), dev(np.ones((V, 3), np.float32))
        dx.copy_(torch.from_numpy(x))
        rc = entries.lc_solve_collisions(_vp(dx), _vp(dxp), _vp(v), _vp(fixed), V, _vp(r), C.c_uint64(300),
                                         C.c_void_p(r.data_ptr() + 300 * 48), C.c_uint64(contacts - 300), *prm, None)
        torch.cuda.synchronize()
        return rc, torch.equal(dx.cpu(), torch.from_numpy(x)) and bool((v == 1).all())

    entries.set_give_up(0)
    assert call(rec) == (0, False)
    bad = rec.copy()
    bad[700, 2] = V
    assert call(bad) == (INVALID, True)
    entries.set_give_up(1)
    assert call(rec) == (TIMEOUT, True)  # and nothing written
    entries.set_give_up(0)
    assert call(rec) == (0, False)


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
