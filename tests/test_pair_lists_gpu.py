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
