"""Triangle bending does not depend on the cloth's place in a batch: its rest
heights, kept beside vertex ids that are shifted by the vertices before the
cloth, are those of the cloth alone."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, scenes
from oracle.parity import run_parity

pytestmark = pytest.mark.gpu


def _bending():
    s = scenes.small_cloth(seed=12, n=28)
    s.params.useTriangleBending = 1
    return s


@pytest.mark.parametrize("variant", [1, 2, 3])
def test_behind_a_large_cloth(cuda, variant):
    spec = _bending()
    before = scenes.small_cloth(seed=1, n=128, thickness=0.3 / 128)
    states = []
    for specs in ([spec], [before, spec]):
        with ClothBatch(specs, solver_variant=variant) as b:
            b.step(30)
            b.sync()
            states.append(b.get_state(len(specs) - 1))
    for k in ("x", "x_prev", "v"):
        assert np.array_equal(states[0][k].view(np.uint32), states[1][k].view(np.uint32)), k


@pytest.mark.parametrize("variant", [1, 2, 3])
def test_parity_behind_a_dihedral_cloth(cuda, variant):
    run_parity([scenes.small_cloth(seed=13, n=16), _bending()], steps=40, check_every=10, variant=variant)
