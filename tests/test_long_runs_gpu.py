"""63-bit codes whose top halves are equal in long runs, in segments that the
general passes sort: the order is a stable sort by the whole code (numpy's)
for runs around every size at which the way a run is finished changes, and the
time does not depend on the codes."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, Lbvh, scenes
from oracle import parity
from oracle.oracle_ffi import Oracle

pytestmark = pytest.mark.gpu

CELL = 1.0 / 1024  # of the top half: ten or eleven of the 21 bits of each axis

RUNS = {
    "rank_limit": [1, 2, 63, 64, 65, 66, 67],
    "counted": [65, 300, 511, 512, 513],
    "one_tile": [513, 700, 2047, 2048, 2049],
    "tiles": [2049, 4096, 4097, 10_000],
    "mixed": [1, 64, 65, 512, 513, 2048, 2049, 6000, 30_000],
    "one": [1 << 30],
}


def _boxes(lengths, n: int, kind: str, rng):
    """n boxes in cells of the given numbers of boxes, in random order.  kind:
    the codes within a cell are spread, of two values, equal, or in order."""
    reps = np.resize(np.minimum(lengths, n), n)
    reps = reps[: int(np.searchsorted(np.cumsum(reps), n)) + 1]
    cell = np.repeat(np.arange(len(reps)), reps)[:n]
    corner = rng.permutation(1023 ** 2)[: cell[-1] + 1]
    p = np.stack([corner % 1023, corner // 1023, np.full(len(corner), 400)], 1)[cell] * CELL
    if kind == "two":
        p = p + 1e-5 + rng.integers(0, 2, (n, 1)) * 4e-6
    elif kind == "spread":
        p = p + rng.uniform(1e-5, 0.4 * CELL, (n, 3))
    else:
        p = p + 1e-5
    p = p[rng.permutation(n)]
    half = np.float32(2.0 ** -10)
    q = p.astype(np.float32)
    return np.ascontiguousarray(q - half), np.ascontiguousarray(q + half)


def _codes(lo, hi):
    mid = lo + (hi - lo) / np.float32(2)
    q = np.clip(mid * np.float32(2097152), np.float32(0), np.float32(2097151)).astype(np.uint64)
    code = np.zeros(len(lo), np.uint64)
    for b in range(21):
        for ax in range(3):
            code |= ((q[:, ax] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - ax)
    return code


def _longest(code):
    _, counts = np.unique(code >> np.uint64(32), return_counts=True)
    return int(counts.max())


@pytest.mark.parametrize("n", [32_769, 40_961, 131_073])
@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("kind", ["spread", "two", "equal"])
def test_order(cuda, n, runs, kind):
    torch = cuda
    lo, hi = _boxes(RUNS[runs], n, kind, np.random.default_rng([n, len(runs)]))
    code = _codes(lo, hi)
    assert _longest(code) > 64
    tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    order = np.argsort(code, kind="stable")
    h = Lbvh(n)
    try:
        for _ in range(2):  # the second sort starts from cleared counts
            h.build(tl.data_ptr(), th.data_ptr(), n)
            assert np.array_equal(h.debug("PERM"), order.astype(np.uint32))
            assert np.array_equal(h.debug("MORTON"), code[order])
    finally:
        h.close()


def _clamped(n: int, seed: int):
    """A cloth around the origin of a Morton frame that begins there: in most
    of it one or two coordinates clamp."""
    s = scenes.small_cloth(seed=seed, n=n, thickness=0.3 / n)
    s.params.worldMin[:] = (-2.0, -2.0, -2.0)
    s.positions -= np.float32([0.5, 1.0, 0.9])
    return s


@pytest.mark.parametrize("sides", [[34, 45], [47, 64], [65, 80, 20]], ids=["4096", "8192", "general"])
def test_batches(cuda, sides):
    """Nine cloths and more: segments of up to 4096 and 8192 keys in one CTA each, and the general passes."""
    specs = [_clamped(sides[k % len(sides)], k) for k in range(10)]
    with ClothBatch(specs, debug_capture=True) as b:
        pre = [b.get_state(c)["vn"] for c in range(len(specs))]
        b.step(1)
        b.sync()
        for c in (0, 1, 2, 9):
            assert _longest(b.debug(c, "MORTON")) > 64
            o32 = Oracle([specs[c]], fp64=False)
            try:
                parity.check_collision(b, c, o32, pre[c], tag=f"cloth {c}")
            finally:
                o32.close()


@pytest.mark.parametrize("kind", ["spread", "two"])
def test_time_does_not_depend_on_the_codes(cuda, kind):
    """A million boxes of one cell of the top half against a million spread
    over the cube.  Twice the passes are expected, 64 times the time was taken
    when one block sorted a run; the bound is 3."""
    torch = cuda
    n = 1_000_000
    rng = np.random.default_rng(0)
    spread = scenes.random_triangle_boxes(n)
    us = []
    h = Lbvh(n)
    try:
        for lo, hi in (spread, _boxes([n], n, kind, rng)):
            tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
            times = []
            for _ in range(9):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record()
                h.build(tl.data_ptr(), th.data_ptr(), n, torch.cuda.current_stream())
                b.record()
                torch.cuda.synchronize()
                times.append(a.elapsed_time(b))
            us.append(float(np.median(times)))
    finally:
        h.close()
    assert us[1] < 3 * us[0], us
