"""Stiffnesses given as device arrays against the same values from the host,
and reverse steps whose gradients live in other buffers each time."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from licenta_gb300 import ClothBatch, _ffi, scenes
from licenta_gb300.adjoint import DiffCloth

pytestmark = pytest.mark.gpu


def _set(batch, ks, kb, host: bool) -> None:
    p = lambda a: None if a is None else C.c_void_p(a.data_ptr())  # noqa: E731
    _ffi.check(_ffi.lib().lc_batch_set_constraint_stiffness(batch._h, p(ks), p(kb), 1 if host else 0), "set")


@pytest.mark.parametrize("which", ["both", "stretch", "bend"])
def test_device_stiffness_equals_host_stiffness(cuda, which):
    """The device's pow may differ from the host's in the last bits of a
    double, so a converted value by one float rounding (6e-8 of it), which
    moves a vertex by less than 1e-8 m an iteration."""
    specs = [scenes.small_cloth(seed=1, n=9), scenes.small_cloth(seed=2, n=20, iterations=7)]
    states = []
    for host in (True, False):
        with ClothBatch(specs) as b:
            counts = [b.constraint_counts(c) for c in range(2)]
            rng = np.random.default_rng(0)
            ks, kb = (torch.from_numpy(rng.uniform(0.0, 1.0, sum(n)).astype(np.float32)) for n in zip(*counts))
            ks[0], ks[1], kb[0] = 0.0, 1.0, 1.0
            ks, kb = (ks if which != "bend" else None), (kb if which != "stretch" else None)
            if not host:
                ks, kb = (None if t is None else t.cuda() for t in (ks, kb))
            _set(b, ks, kb, host)
            b.step(3)
            b.sync()
            states.append([b.get_state(c)["x"] for c in range(2)])
    for h, d in zip(*states):
        assert np.abs(h - d).max() < 1e-6


@pytest.mark.parametrize("stiffness,rescaled", [(True, True), (True, False), (False, False)])
def test_reverse_step_does_not_depend_on_the_buffers(cuda, stiffness, rescaled):
    cloth = DiffCloth([scenes.adjoint_cloth(n=12), scenes.adjoint_cloth(n=17)])
    gen = torch.Generator(device="cuda").manual_seed(3)
    seed = [torch.randn((cloth.V, 3), generator=gen, device="cuda") for _ in range(3)]
    kseed = [torch.randn(n, generator=gen, device="cuda") for n in (cloth.E, cloth.B)]
    results, held = [], []
    for _ in range(3):
        cloth.load(cloth.initial)
        g = [t.clone() for t in seed] + ([t.clone() for t in kseed] if stiffness else [None, None])
        e = torch.zeros(2, dtype=torch.int32, device="cuda") if rescaled else None
        cloth.adjoint_step(*g, e)
        torch.cuda.synchronize()
        results.append([t.cpu().numpy().view(np.uint32) for t in g if t is not None])
        held.append(g)  # the next pass gets other addresses
    if stiffness:
        assert all(np.abs(t.cpu().numpy() - s.cpu().numpy()).max() > 0 for t, s in zip(held[0][3:], kseed))
    for r in results[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(r, results[0]))
