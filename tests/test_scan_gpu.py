"""The device-wide scan at the edges of its tiles and of its largest grid,
through the sweep-and-prune broadphase (one count per object): boxes in a row,
each touching the next, give the pairs (i, i + 1) in order."""
from __future__ import annotations

import pytest
import torch

from licenta_gb300.broadphase import Broadphase

pytestmark = pytest.mark.gpu

TILE, GRID = 4096, 304


@pytest.mark.parametrize("n", [1, 2, 257, TILE - 1, TILE, TILE + 1, 3 * TILE + 17, GRID * TILE - 1, GRID * TILE + 1,
                               2 * GRID * TILE + 5])
def test_row_of_boxes(cuda, n):
    i = torch.arange(n, dtype=torch.float32, device="cuda")  # exact below 2^24
    lo = torch.stack([i, torch.zeros_like(i), torch.zeros_like(i)], dim=1)
    bp = Broadphase("sap", n)
    for hi_x in (1.0, 0.5):  # touching, then apart: the same handle's second scan starts from cleared sums
        hi = lo + torch.tensor([hi_x, 1.0, 1.0], device="cuda")
        bp.update(lo, hi)
        pairs = bp.test()
        k = torch.arange(n - 1 if hi_x == 1.0 else 0, device="cuda")
        assert torch.equal(pairs, torch.stack([k, k + 1], dim=1))
    bp.close()
