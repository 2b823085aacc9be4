"""Small cloths between cloths whose hierarchy is malformed (three equal Morton
codes meet), in one block of slots of the hierarchy kernel: every cloth's codes,
tree, boxes, pairs and contacts are the oracle's, on the first step, when no
earlier step has left anything in the node records, and after the next."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, scenes
from oracle import parity
from oracle.oracle_ffi import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", [[5], [2, 3], [6, 4]])
def test_small_cloths_between_flagged_ones(cuda, between):
    flagged = [scenes.equal_code_cloth(seed=26 + k) for k in range(2)]
    small = [scenes.small_cloth(seed=n, n=n, thickness=0.3 / n) for n in between]
    # more than one sort tile: the kernel whose blocks hold slots of several cloths
    specs = [flagged[0], *small, flagged[1], scenes.small_cloth(seed=9, n=40, thickness=0.3 / 40)]
    first = sum(s.num_triangles for s in specs[:-2])
    assert first < 256 < first + specs[-2].num_triangles  # the first block begins and ends in flagged cloths
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
                if step == 0:
                    m = np.sort(b.debug(c, "MORTON"))
                    assert bool((m[2:] == m[:-2]).any()) == (c in (0, len(specs) - 2)), c
