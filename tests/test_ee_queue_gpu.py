"""Edge-edge candidates whose edges are apart throughout their times' advances
skip the tests, and the others are tested 32 at a time: the contacts of
random triangle pairs, over sizes, speeds, thicknesses and distances from the
origin, bit for bit those of the oracle, which tests every candidate."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle_ffi import narrow_contacts

pytestmark = pytest.mark.gpu


def _soup(rng, pairs: int, edge: float, offset: float, speed: float, kind: str):
    """Pairs of triangles about one edge apart, moving at up to `speed` edges
    per step (dt = 1/64)."""
    c = rng.uniform(-1, 1, (pairs, 1, 3)) * edge * 20 + offset
    t = rng.normal(0, 1, (pairs, 6, 3)) * edge * 0.5
    if kind == "flat":  # coplanar pairs
        t[..., 1] = 0
    if kind == "parallel":  # the second triangle a moved copy of the first
        t[:, 3:] = t[:, :3] + rng.normal(0, 0.3, (pairs, 1, 3)) * edge
    if kind == "degenerate":  # edges of no length
        t[::2, 1] = t[::2, 0]
        t[1::3, 4] = t[1::3, 3]
    x = (c + t).reshape(-1, 3).astype(np.float32)
    v = (rng.normal(0, 1, (pairs, 6, 3)) * 0.3 + rng.normal(0, 1, (pairs, 1, 3))).reshape(-1, 3) * speed * edge * 64
    v[rng.random(len(v)) < 0.2] = 0
    v = v.astype(np.float32)
    return x, v


@pytest.mark.parametrize("pairs", [1, 5, 700])
@pytest.mark.parametrize("kind", ["free", "flat", "parallel", "degenerate"])
@pytest.mark.parametrize("edge,offset", [(0.01, 0.0), (0.02, 3.0), (1.0, 100.0), (0.05, 3000.0)])
@pytest.mark.parametrize("thick,speed", [(0.0, 0.5), (0.02, 0.0), (0.3, 0.1), (0.3, 3.0), (4.0, 0.5)])
def test_contacts_equal_the_oracle(cuda, pairs, kind, edge, offset, thick, speed):
    torch = cuda
    from licenta_gb300 import Narrowphase
    rng = np.random.default_rng([pairs, len(kind), int(offset), int(10 * thick), int(10 * speed)])
    xp, v = _soup(rng, pairs, edge, offset, speed, kind)
    dt, h = np.float32(1 / 64), np.float32(thick * edge)
    x = xp + v * dt
    tris = np.arange(6 * pairs, dtype=np.uint32).reshape(-1, 3)
    feats = np.full(2 * pairs, 0x3F, np.uint8)
    pr = np.arange(2 * pairs, dtype=np.uint32).reshape(-1, 2)
    want = narrow_contacts(0, x, xp, v, tris, feats, pr, float(h), float(dt))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dx, dxp, dv, dtr, df, dp = dev(x), dev(xp), dev(v), dev(tris), dev(feats), dev(pr)
    cap = 15 * pairs
    out = [torch.zeros((cap, 12), dtype=torch.int32, device="cuda") for _ in range(2)]
    n = Narrowphase(len(xp), 2 * pairs, pairs)
    try:
        rc, nvf, nee = n.run(dx.data_ptr(), dxp.data_ptr(), dv.data_ptr(), len(xp), dtr.data_ptr(), df.data_ptr(),
                             2 * pairs, dp.data_ptr(), pairs, float(h), float(dt), out[0].data_ptr(), cap,
                             out[1].data_ptr(), cap)
    finally:
        n.close()
    assert rc == 0
    for got, cnt, ref in ((out[0], nvf, want[0]), (out[1], nee, want[1])):
        assert cnt == len(ref)
        g, r = got[:cnt].cpu().numpy(), np.ascontiguousarray(ref).view(np.int32).reshape(cnt, 12)
        both_nan = np.isnan(g.view(np.float32)) & np.isnan(r.view(np.float32))  # (a NaN's payload is the processor's)
        assert np.array_equal(g[~both_nan], r[~both_nan])


def test_many_pairs_equal_the_same_pairs_few_at_a_time(cuda):
    """More pairs than the rule gives one launch for both kinds: the contacts
    of a repeated list are the list's, repeated."""
    torch = cuda
    from licenta_gb300 import Narrowphase
    rng = np.random.default_rng(9)
    pairs, reps = 700, 710
    xp, v = _soup(rng, pairs, 0.02, 0.0, 0.5, "free")
    dt, h = 1 / 64, 0.3 * 0.02
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dx, dxp, dv = dev(xp + v * np.float32(dt)), dev(xp), dev(v)
    dtr = dev(np.arange(6 * pairs, dtype=np.uint32).reshape(-1, 3))
    df = dev(np.full(2 * pairs, 0x3F, np.uint8))
    pr = np.arange(2 * pairs, dtype=np.uint32).reshape(-1, 2)

    def run(p):
        cap = 2 * len(p)
        out = [torch.zeros((cap, 12), dtype=torch.int32, device="cuda") for _ in range(2)]
        n = Narrowphase(len(xp), 2 * pairs, len(p), candidate_capacity=15 * len(p), contact_capacity=cap)
        try:
            dp = dev(p)
            rc, nvf, nee = n.run(dx.data_ptr(), dxp.data_ptr(), dv.data_ptr(), len(xp), dtr.data_ptr(), df.data_ptr(),
                                 2 * pairs, dp.data_ptr(), len(p), h, dt, out[0].data_ptr(), cap, out[1].data_ptr(), cap)
        finally:
            n.close()
        assert rc == 0
        return out[0][:nvf].cpu().numpy(), out[1][:nee].cpu().numpy()

    few, many = run(pr), run(np.tile(pr, (reps, 1)))
    for a, b in zip(few, many):
        assert len(a) > 50
        assert np.array_equal(np.tile(a, (reps, 1)), b)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("vertices,triangles", [(4, 6), (9, 40), (30, 33)])
def test_ownership_and_shared_vertices(cuda, mode, vertices, triangles):
    """Triangles with zero to three vertices in common, every ownership byte."""
    torch = cuda
    from licenta_gb300 import Narrowphase, _ffi
    rng = np.random.default_rng([vertices, mode])
    xp = rng.uniform(0, 0.05, (vertices, 3)).astype(np.float32)
    v = rng.normal(0, 1, (vertices, 3)).astype(np.float32)
    x = xp + v * np.float32(1 / 64)
    tris = np.stack([rng.permutation(vertices)[:3] for _ in range(triangles)]).astype(np.uint32)
    feats = rng.integers(0, 64, triangles).astype(np.uint8)
    a, b = np.triu_indices(triangles, 1)
    pr = np.stack([a, b], 1).astype(np.uint32)
    h, dt = 0.01, 1 / 64
    want = narrow_contacts(mode, x, xp, v, tris, feats, pr, h, dt)
    dev = lambda q: torch.from_numpy(np.ascontiguousarray(q)).cuda()
    dx, dxp, dv, dtr, df, dp = dev(x), dev(xp), dev(v), dev(tris), dev(feats), dev(pr)
    cap = 15 * len(pr)
    out = [torch.zeros((cap, 12), dtype=torch.int32, device="cuda") for _ in range(2)]
    n = Narrowphase(vertices, triangles, len(pr), candidate_capacity=cap, contact_capacity=cap)
    try:
        rc, nvf, nee = n.run(dx.data_ptr(), dxp.data_ptr(), dv.data_ptr(), vertices, dtr.data_ptr(), df.data_ptr(),
                             triangles, dp.data_ptr(), len(pr), h, dt, out[0].data_ptr(), cap, out[1].data_ptr(), cap,
                             mode=_ffi.LC_NARROW_DCD if mode else _ffi.LC_NARROW_CCD)
    finally:
        n.close()
    assert rc == 0 and (vertices == 4 or len(want[1]) > 0)  # (four vertices leave one disjoint edge per edge)
    for got, cnt, ref in ((out[0], nvf, want[0]), (out[1], nee, want[1])):
        assert cnt == len(ref)
        g, r = got[:cnt].cpu().numpy(), np.ascontiguousarray(ref).view(np.int32).reshape(cnt, 12)
        both_nan = np.isnan(g.view(np.float32)) & np.isnan(r.view(np.float32))
        assert np.array_equal(g[~both_nan], r[~both_nan])
