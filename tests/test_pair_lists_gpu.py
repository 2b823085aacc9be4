"""Pair and contact lists built by several lanes: leaves with 0 to a full chunk
of pairs, around the lanes per leaf; contact lists in contact order whatever
order their entries arrived in."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, Lbvh, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1, 7, 8, 9, 16, 64])
@pytest.mark.parametrize("n", [2, 9, 33, 70, 300])
def test_leaf_pairs(cuda, n, chunk):
    """n overlapping boxes: leaf i pairs with its first min(chunk, n - 1 - i) successors."""
    torch = cuda
    rng = np.random.default_rng(n)
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    lo, hi = torch.from_numpy(c - 2).cuda(), torch.from_numpy(c + 2).cuda()
    t = Lbvh(n, chunk_size=chunk)
    try:
        t.build(lo.data_ptr(), hi.data_ptr(), n)
        out = torch.full((n * chunk + 1, 2), -1, dtype=torch.int32, device="cuda")
        got = t.pairs(out.data_ptr(), n * chunk)
        p = out[:got].cpu().numpy()
        assert len(set(t.debug("MORTON").tolist())) == n  # (three equal codes can hide leaves)
        want = np.minimum(chunk, n - 1 - np.arange(n))
        assert got == want.sum()
        order = p[:, 0]
        # runs of one first index, of the leaves' lengths
        if got:
            starts = np.flatnonzero(np.r_[True, order[1:] != order[:-1]])
            assert np.array_equal(np.diff(np.r_[starts, got]), want[want > 0])
            assert len({tuple(sorted(q)) for q in p.tolist()}) == got
    finally:
        t.close()


@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 33])
def test_many_leaves(cuda, n):
    """Around the size at which a warp takes 32 leaves: a chain of boxes, each
    overlapping the next one along x, pairs with and without gaps."""
    torch = cuda
    k = np.arange(n, dtype=np.float64)
    lo = np.stack([k / n, np.zeros(n), np.zeros(n)], 1)
    hi = lo + [[1.4 / n, 1e-3, 1e-3]]
    hi[::3, 0] = lo[::3, 0] + 0.4 / n  # every third reaches nobody
    lo, hi = lo.astype(np.float32), hi.astype(np.float32)
    want = {(i, i + 1) for i in np.flatnonzero(hi[:-1, 0] >= lo[1:, 0]).tolist()}
    t = Lbvh(n)
    try:
        dl, dh = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
        t.build(dl.data_ptr(), dh.data_ptr(), n)
        out = torch.zeros((4 * n, 2), dtype=torch.int32, device="cuda")
        got = t.pairs(out.data_ptr(), 4 * n)
        ids = torch.zeros(n, dtype=torch.int32, device="cuda")
        t.sorted_ids(ids.data_ptr())
        ids = ids.cpu().numpy()
        p = out[:got].cpu().numpy()
    finally:
        t.close()
    assert np.all(np.diff(p[:, 0]) >= 0)
    pairs = np.sort(ids[p], axis=1)
    overlap = hi[pairs[:, 0], 0] >= lo[pairs[:, 1], 0]
    assert overlap.all() and len({tuple(q) for q in pairs.tolist()}) == got
    assert want <= {tuple(q) for q in pairs.tolist()}


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("friction", [0, 1])
def test_contact_lists_are_ordered(cuda, variant, friction):
    """Float sums in list order: the same bits on every run."""
    spec = scenes.small_cloth(seed=5, n=48, thickness=1.2 / 48)
    spec.params.useFriction = friction
    p = spec.positions
    p[:, 1] += 0.3 * np.abs(p[:, 2] - p[:, 2].mean())  # creased: layers in reach of each other
    runs = []
    for _ in range(3):
        with ClothBatch([spec], solver_variant=variant, vf_capacity=1 << 19, ee_capacity=1 << 20) as b:
            b.step(3)
            b.sync()
            runs.append((b.get_state(0)["x"].copy(), b.counters()))
    assert runs[0][1]["vf"] + runs[0][1]["ee"] > 1000
    for x, c in runs[1:]:
        assert c == runs[0][1]
        assert np.array_equal(x.view(np.uint32), runs[0][0].view(np.uint32))
