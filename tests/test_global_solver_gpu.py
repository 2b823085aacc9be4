"""The global-memory solver's two forms, tiles and (where a vertex has more
constraints than a tile holds) two launches, against the on-chip solver: the
bound is that of the parity tests, 1e-5 m, whatever the order of the vertices
and the fill of the last tile."""
from __future__ import annotations

import numpy as np
import pytest

from licenta_gb300 import ClothBatch, scenes

pytestmark = pytest.mark.gpu


def _states(specs, variant: int, steps: int):
    with ClothBatch(specs, solver_variant=variant) as b:
        b.step(steps)
        b.sync()
        return [b.get_state(c)["x"] for c in range(len(specs))]


def _compare(specs, steps: int = 2):
    for got, want in zip(_states(specs, 1, steps), _states(specs, 3, steps)):
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() < 1e-5


def _shuffled(spec, seed):
    p = np.random.default_rng(seed).permutation(len(spec.positions))
    inv = np.argsort(p).astype(np.uint32)
    return scenes.ClothSpec(spec.positions[p], inv[spec.indices], spec.pinned[p], spec.params, spec.meta)


@pytest.mark.parametrize("side", [2, 8, 9, 57, 140, 175])
@pytest.mark.parametrize("shuffle", [False, True])
def test_tiles(cuda, side, shuffle):
    spec = scenes.small_cloth(seed=side, n=side, thickness=0.3 / side)
    _compare([_shuffled(spec, side) if shuffle else spec])


def test_tiles_of_several_cloths(cuda):
    specs = [scenes.small_cloth(seed=n, n=n, thickness=0.3 / n) for n in (5, 40, 23, 71)]
    for s, it in zip(specs, (10, 3, 7, 10)):
        s.params.solverIterations = it
    specs[1].params.useTriangleBending = 1
    _compare(specs)


@pytest.mark.parametrize("spokes", [600, 1500])
def test_a_vertex_of_more_constraints_than_a_tile_holds(cuda, spokes):
    """A fan, away from the origin (the bends take planes through it)."""
    a = np.arange(spokes) * (2 * np.pi / spokes)
    rim = np.stack([0.7 + 0.4 * np.cos(a), 1.5 + 0.02 * np.sin(3 * a), 0.7 + 0.4 * np.sin(a)], 1)
    k = np.arange(spokes, dtype=np.uint32)
    tri = np.stack([np.zeros(spokes, np.uint32), 1 + k, 1 + (k + 1) % spokes], 1)
    base = scenes.small_cloth(n=4, iterations=4, stiffness=0.3, thickness=1e-5)
    _compare([scenes.ClothSpec(np.concatenate([[[0.7, 1.5, 0.7]], rim]).astype(np.float32), tri,
                               np.zeros(spokes + 1, base.pinned.dtype), base.params)], steps=1)
