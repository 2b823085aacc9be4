"""Edge-edge candidates whose first vertex rests in the origin while the other
edge comes from far away within the step and passes at the thickness, give or
take the roundings of its path: the contacts are, bit for bit, those of the
oracle, which tests every candidate."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle_ffi import narrow_contacts

pytestmark = pytest.mark.gpu


def _passing(rng, n: int, h: float, far: float):
    """Triangle A at rest, its first vertex in the origin; B's first vertex
    crosses A's plane `far` metres from where it was, beside A's first edge.
    The midpoints of the two edges face each other across the gap."""
    a = rng.uniform(0, 2 * np.pi, n)
    d, out = np.stack([np.cos(a), 0 * a, np.sin(a)], 1), np.stack([-np.sin(a), 0 * a, np.cos(a)], 1)
    A = np.stack([0 * d, 0.5 * d, 0.25 * d - 0.3 * out], 1)
    gap = h + rng.uniform(0, 2e-3 * h + 4e-7 * far, n)[:, None]
    b0 = 0.2 * d + gap * out
    B = np.stack([b0, b0 + 0.3 * out + 0.1 * d, b0 + 0.3 * out - 0.1 * d], 1)
    m = rng.normal(0, 1, (n, 1, 3))
    m *= far / np.linalg.norm(m, axis=2, keepdims=True)
    m[..., 1] = 0.2
    t = rng.uniform(0.3, 0.7, n)[:, None, None]
    v = np.zeros((n, 6, 3))
    v[:, 3:] = m
    return np.concatenate([A, B - m * t], 1).reshape(-1, 3).astype(np.float32), v.reshape(-1, 3).astype(np.float32)


@pytest.mark.parametrize("far,h", [(1.0, 0.01), (100.0, 0.01), (1000.0, 0.01), (3000.0, 0.05)])
def test_contacts_equal_the_oracle(cuda, far, h):
    torch = cuda
    from licenta_gb300 import Narrowphase
    pairs, dt = 20_000, 1.0
    xp, v = _passing(np.random.default_rng(1), pairs, h, far)
    x = xp + v * np.float32(dt)
    tris = np.arange(6 * pairs, dtype=np.uint32).reshape(-1, 3)
    feats = np.full(2 * pairs, 0x3F, np.uint8)
    pr = np.arange(2 * pairs, dtype=np.uint32).reshape(-1, 2)
    want = narrow_contacts(0, x, xp, v, tris, feats, pr, h, dt)
    assert len(want[1]) >= 20
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dx, dxp, dv, dtr, df, dp = dev(x), dev(xp), dev(v), dev(tris), dev(feats), dev(pr)
    cap = 15 * pairs
    out = [torch.zeros((cap, 12), dtype=torch.int32, device="cuda") for _ in range(2)]
    n = Narrowphase(len(xp), 2 * pairs, pairs, candidate_capacity=cap, contact_capacity=cap)
    try:
        rc, nvf, nee = n.run(dx.data_ptr(), dxp.data_ptr(), dv.data_ptr(), len(xp), dtr.data_ptr(), df.data_ptr(),
                             2 * pairs, dp.data_ptr(), pairs, h, dt, out[0].data_ptr(), cap, out[1].data_ptr(), cap)
    finally:
        n.close()
    assert rc == 0
    for got, cnt, ref in ((out[0], nvf, want[0]), (out[1], nee, want[1])):
        assert cnt == len(ref)
        g, r = got[:cnt].cpu().numpy(), np.ascontiguousarray(ref).view(np.int32).reshape(cnt, 12)
        both_nan = np.isnan(g.view(np.float32)) & np.isnan(r.view(np.float32))
        assert np.array_equal(g[~both_nan], r[~both_nan])
