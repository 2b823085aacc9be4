"""The standalone LBVH's sort and node boxes where their paths meet: segments
around the one-block sort's sizes and the general sort's tiles, with keys whose
top halves tie in short and long runs, and equal codes.  The order is a stable
sort by code (numpy's), the boxes are unions of their children's, and the
pairs are the allocation-free entry's, which climbs the hierarchy instead."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from licenta_gb300 import Lbvh, _ffi

pytestmark = pytest.mark.gpu


def _boxes(kind: str, n: int):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        p = rng.uniform(0.0, 1.0, (n, 3))
    elif kind == "cell":        # every code shares its top half
        p = 0.5 + rng.uniform(0.0, 4e-4, (n, 3))
    elif kind == "clusters":    # runs of about 60 around the one-by-one limit
        p = rng.uniform(0.0, 1.0, (max(1, n // 60), 3))[rng.integers(0, max(1, n // 60), n)]
        p = np.floor(p * 1024) / 1024 + rng.uniform(0.0, 9e-4, (n, 3))
    elif kind == "pairs":       # every code twice
        p = np.repeat(rng.uniform(0.0, 1.0, ((n + 1) // 2, 3)), 2, axis=0)[rng.permutation(2 * ((n + 1) // 2))[:n]]
    else:                       # few distinct codes, many times each
        p = rng.uniform(0.0, 1.0, (max(1, n // 40), 3))[rng.integers(0, max(1, n // 40), n)]
    half = rng.uniform(1e-4, 2e-3, (n, 3))
    if kind in ("pairs", "equal"):
        half[:] = 1e-3          # the same box around the same point
    return (p - half).astype(np.float32), (p + half).astype(np.float32)


def _codes(lo, hi, mode):
    mid = lo + (hi - lo) / np.float32(2)
    bits, scale = (10, np.float32(1024)) if mode == _ffi.LC_MORTON_K30 else (21, np.float32(2097152))
    q = np.clip(mid * scale, np.float32(0), scale - np.float32(1)).astype(np.uint64)
    code = np.zeros(len(lo), np.uint64)
    for b in range(bits):
        for ax in range(3):
            code |= ((q[:, ax] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - ax)
    return code


SIZES = [2, 3, 63, 64, 65, 66, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 20011]


@pytest.mark.parametrize("mode", [_ffi.LC_MORTON_REF63, _ffi.LC_MORTON_K30], ids=["ref63", "k30"])
@pytest.mark.parametrize("kind", ["uniform", "cell", "clusters", "pairs", "equal"])
def test_order_and_boxes(cuda, kind, mode):
    h = Lbvh(max(SIZES), chunk_size=64, morton_mode=mode)
    for n in SIZES:
        lo, hi = _boxes(kind, n)
        tl, th = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
        h.build(tl.data_ptr(), th.data_ptr(), n, torch.cuda.current_stream())
        code = _codes(lo, hi, mode)
        order = np.argsort(code, kind="stable")
        assert np.array_equal(h.debug("PERM"), order.astype(np.uint32)), n
        assert np.array_equal(h.debug("MORTON"), code[order]), n
        sorted_code = code[order]
        box = h.debug("NODE_AABB")
        assert np.array_equal(box[n - 1:, :3], lo[order]) and np.array_equal(box[n - 1:, 3:], hi[order]), n
        triple = n > 2 and bool((sorted_code[2:] == sorted_code[:-2]).any())
        if not triple:  # a tree: every node's box, rightmost leaves and parents
            left, right, par, rml = (h.debug(k) for k in ("LEFTS", "RIGHTS", "PARENTS", "RML"))
            assert np.array_equal(box[:n - 1, :3], np.minimum(box[left, :3], box[right, :3])), n
            assert np.array_equal(box[:n - 1, 3:], np.maximum(box[left, 3:], box[right, 3:])), n
            ids = np.arange(n - 1)
            assert np.array_equal(par[left], ids) and np.array_equal(par[right], ids) and par[0] == -1, n
            own = np.concatenate([rml.max(axis=1), np.arange(n - 1, 2 * n - 1)])
            assert np.array_equal(rml[:, 0], own[left]) and np.array_equal(rml[:, 1], own[right]), n
        if n <= 2048:
            cap = 64 * n
            a, b = (torch.zeros((cap, 2), dtype=torch.int32, device="cuda") for _ in range(2))
            k = h.pairs(a.data_ptr(), cap, torch.cuda.current_stream())
            m = C.c_uint64()
            _ffi.check(_ffi.lib().lc_lbvh_pairs_static(
                C.c_void_p(tl.data_ptr()), C.c_void_p(th.data_ptr()), n, 64, mode, C.c_void_p(b.data_ptr()), cap,
                C.byref(m), None, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "lc_lbvh_pairs_static")
            assert k == m.value and torch.equal(a[:k], b[:k]), n
    h.close()
