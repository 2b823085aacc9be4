"""Hierarchies of large segments, bit for bit the oracle's: where three equal
codes meet (the two-pass climb with its record pass, above 8192 leaves), and
the levels of the range tree that only segments of more than a million leaves
have."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, Lbvh, _ffi, scenes
from oracle import parity
from oracle.oracle_ffi import Oracle, lbvh_boxes

pytestmark = pytest.mark.gpu

ARRAYS = ("MORTON", "PERM", "LEFTS", "RIGHTS", "PARENTS", "RML", "NODE_AABB", "PAIRS")


def _boxes(kind: str, n: int):
    rng = np.random.default_rng(n)
    if kind == "triples":      # mostly distinct codes, three equal ones here and there
        p = rng.uniform(0.0, 1.0, (n, 3))
        at = rng.choice(n - 2, n // 50, replace=False)
        p[at + 1] = p[at]
        p[at + 2] = p[at]
    elif kind == "few":        # every code many times
        p = rng.uniform(0.0, 1.0, (max(1, n // 40), 3))[rng.integers(0, max(1, n // 40), n)]
    else:                      # around the frame's origin: one to three coordinates clamp
        p = rng.uniform(-0.7, 0.7, (n, 3)) * [1.0, 0.2, 1.0]
    half = np.float32(2e-3)
    q = p.astype(np.float32)
    return q - half, q + half


@pytest.mark.parametrize("mode", [_ffi.LC_MORTON_REF63, _ffi.LC_MORTON_K30], ids=["ref63", "k30"])
@pytest.mark.parametrize("kind", ["triples", "few", "clamped"])
def test_flagged_segment(cuda, kind, mode):
    torch = cuda
    sizes = [70_001, 32_769, 16_385, 8_193]
    h = Lbvh(max(sizes), 64, mode)
    try:
        for n in sizes:
            lo, hi = _boxes(kind, n)
            want = lbvh_boxes(lo, hi, chunk=64, mode=mode)
            m = want["MORTON"]
            assert (m[2:] == m[:-2]).any()
            tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
            h.build(tl.data_ptr(), th.data_ptr(), n)
            count = h.pairs(None, 0)
            for what in ARRAYS:
                got, exp = h.debug(what), want[what]
                if what == "NODE_AABB":
                    got, exp = got.view(np.uint32), exp.view(np.uint32)
                assert got.shape == exp.shape and np.array_equal(got, exp), (n, what)
            assert count == len(want["PAIRS"]), n
    finally:
        h.close()


def test_flagged_and_plain_cloths_in_one_batch(cuda):
    """Blocks of the climb that hold slots of flagged and of other cloths; a
    cloth of more than 8192 triangles makes the batch take the two passes."""
    specs = [scenes.equal_code_cloth(seed=26), scenes.small_cloth(seed=2, n=70, thickness=0.3 / 70),
             scenes.equal_code_cloth(seed=27), scenes.small_cloth(seed=3, n=9, thickness=0.3 / 9)]
    with ClothBatch(specs, debug_capture=True) as b:
        for step in range(2):
            pre = [b.get_state(c)["vn"] for c in range(len(specs))]
            b.step(1)
            b.sync()
            for c, s in enumerate(specs):
                o32 = Oracle([s], fp64=False)
                try:
                    parity.check_collision(b, c, o32, pre[c], tag=f"step {step}, cloth {c}")
                finally:
                    o32.close()


@pytest.mark.parametrize("n", [(1 << 20) + 1, (1 << 21) + 4099])
def test_more_than_a_million_leaves(cuda, n):
    """Every node's box is the union of its children's."""
    torch = cuda
    lo, hi = scenes.random_triangle_boxes(n, seed=n)
    tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    h = Lbvh(n, 4)
    try:
        h.build(tl.data_ptr(), th.data_ptr(), n)
        order, box, left, right, par = (h.debug(k) for k in ("PERM", "NODE_AABB", "LEFTS", "RIGHTS", "PARENTS"))
        m = h.debug("MORTON")
    finally:
        h.close()
    assert not (m[2:] == m[:-2]).any()
    assert np.array_equal(box[n - 1:, :3], lo[order]) and np.array_equal(box[n - 1:, 3:], hi[order])
    assert np.array_equal(box[:n - 1, :3], np.minimum(box[left, :3], box[right, :3]))
    assert np.array_equal(box[:n - 1, 3:], np.maximum(box[left, 3:], box[right, 3:]))
    ids = np.arange(n - 1)
    assert np.array_equal(par[left], ids) and np.array_equal(par[right], ids) and par[0] == -1


@pytest.mark.parametrize("kind", ["triples", "few", "clamped"])
def test_flagged_segment_of_one_launch(cuda, kind):
    """Up to 8192 leaves: one block per cloth, or a cluster of eight."""
    torch = cuda
    h = Lbvh(8192)
    try:
        for n in (8192, 8191, 4097, 2049, 2048, 1025, 1024, 70):
            lo, hi = _boxes(kind, n)
            want = lbvh_boxes(lo, hi, chunk=64, mode=_ffi.LC_MORTON_REF63)
            tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
            h.build(tl.data_ptr(), th.data_ptr(), n)
            count = h.pairs(None, 0)
            for what in ARRAYS:
                got, exp = h.debug(what), want[what]
                if what == "NODE_AABB":
                    got, exp = got.view(np.uint32), exp.view(np.uint32)
                assert got.shape == exp.shape and np.array_equal(got, exp), (n, what)
            assert count == len(want["PAIRS"]), n
    finally:
        h.close()


@pytest.mark.parametrize("count", [3, 9])
def test_flagged_cloths_of_up_to_8192_triangles(cuda, count):
    """Few cloths (clusters) and more (three launches), some of them clamped at the frame's faces."""
    specs = []
    for k in range(count):
        s = scenes.small_cloth(seed=k, n=(64, 40, 12)[k % 3], thickness=0.1 / 64)
        if k % 2 == 0:
            s.params.worldMin[:] = (-2.0, -2.0, -2.0)
            s.positions -= np.float32([0.5, 1.0, 0.9])
        specs.append(s)
    with ClothBatch(specs, debug_capture=True) as b:
        for step in range(2):
            pre = [b.get_state(c)["vn"] for c in range(count)]
            b.step(1)
            b.sync()
            flagged = 0
            for c, s in enumerate(specs):
                m = b.debug(c, "MORTON")
                flagged += bool((m[2:] == m[:-2]).any())
                o32 = Oracle([s], fp64=False)
                try:
                    parity.check_collision(b, c, o32, pre[c], tag=f"step {step}, cloth {c}")
                finally:
                    o32.close()
            assert 0 < flagged < count
