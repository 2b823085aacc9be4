"""lc_solve_collisions with vertices in many contacts: every vertex sums its
impulses in contact order, whatever order its list was filled in, so runs give
the same bits, those of the oracle's sums."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from licenta_gb300 import _ffi
from oracle.oracle_ffi import solve_collisions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vertices,contacts", [(4, 1), (4, 64), (9, 257), (40, 5000)])
def test_sums_in_contact_order(cuda, vertices, contacts):
    torch = cuda
    rng = np.random.default_rng(vertices + contacts)
    x = rng.uniform(0, 1, (vertices, 3)).astype(np.float32)
    xp, v = x - np.float32(0.001), rng.normal(0, 1, (vertices, 3)).astype(np.float32)
    rec = np.zeros((contacts, 12), np.int32)
    rec[:, :4] = np.stack([rng.permutation(vertices)[:4] for _ in range(contacts)])
    f = rec.view(np.float32)
    w = rng.uniform(0.1, 1, (contacts, 4)).astype(np.float32)
    f[:, 4:8] = w / w.sum(1, keepdims=True)
    f[:, 8] = rng.uniform(0, 1, contacts)
    n = rng.normal(0, 1, (contacts, 3))
    f[:, 9:12] = n / np.linalg.norm(n, axis=1, keepdims=True)
    vf, ee = rec[: contacts // 3], rec[contacts // 3:]
    fixed = np.zeros(vertices, np.uint8)
    fixed[0] = 1
    prm = (0.9, 0.01, 1 / 60, 0.02)
    want = solve_collisions(x, xp, v, fixed, vf, ee, stiffness=prm[0], vertex_mass=prm[1], dt=prm[2],
                            thickness=prm[3])
    runs = []
    for _ in range(2):
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        t = [dev(a) for a in (x, xp, v, fixed, vf, ee)]
        vp = lambda q: C.c_void_p(q.data_ptr())
        rc = _ffi.lib().lc_solve_collisions(vp(t[0]), vp(t[1]), vp(t[2]), vp(t[3]), vertices, vp(t[4]) if len(vf) else None,
                                            len(vf), vp(t[5]), len(ee), *prm, None)
        torch.cuda.synchronize()
        assert rc == 0, _ffi.lib().lc_last_error_string()
        runs.append((t[0].cpu().numpy(), t[2].cpu().numpy()))
    for got, again, ref in zip(runs[0], runs[1], want):
        assert np.array_equal(got.view(np.uint32), again.view(np.uint32))
        assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
