"""Timed cases of the framework's public entry points.

Each case is one call, or the few calls, that a program makes again and again:
a step of one cloth or of many, a step with its state on the host, a
differentiable rollout forward and back, the standalone LBVH query, the
collision pipeline a caller composes, and the object-level broadphase.  Sizes
are those of the five workloads of licenta_gb300/scenes.py, of bench.py and of
the tests, and the ranges around them.

Every input is made from the seed alone, in numpy, and never by stepping the
engine: a cloth is created flat (its rest state) and given a state it takes in
a rollout, a sheet swinging about its pinned edge, smooth or folded onto
itself, or one about to land on a sphere.  A stepped batch is put back to that
state at the start of every pass (lc_batch_load_state, as a rollout restarts
from a checkpoint), with the triangle order of the step before.

exact() restates the contact-free step in 64 bits and differentiates it with
torch's autograd.  The cases with self-collision have no 64-bit value: which
contacts exist is decided by the 32-bit arithmetic of the collision stages.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from licenta_gb300 import ClothBatch, ClothBatchGroup, Lbvh, Narrowphase, _ffi, scenes
from licenta_gb300.adjoint import ClothRollout, DiffCloth
from licenta_gb300.broadphase import Broadphase

DT = 1.0 / 60.0


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # the small plain workload: one 32x32 cloth, a few steps of its rollout (launches and latency)
        dict(name="cloth_32", kind="step", n=32, steps=3, fold=False, wind=False, friction=False, tri_bend=False,
             thickness=0.01),
        # one ordinary cloth with the options a scene turns on: wind, friction, folds in contact
        dict(name="cloth_101_folded", kind="step", n=101, steps=1, fold=True, wind=True, friction=True,
             tri_bend=False, thickness=0.0),
        # the large plain workload: 512x512, 20 iterations, landing on the analytic sphere
        dict(name="drop_512", kind="drop", n=512),
        # the batched workload: uneven cloths (side 16..192) in two concurrent lanes, in contact
        dict(name="batch_128", kind="batch", count=128, n_min=16, n_max=192, lanes=2, morton="ref63", tri_bend=False),
        # a smaller batch with its state on the host: copied in, stepped, copied out (with triangle bending)
        dict(name="batch_host_24", kind="host", count=24, n_min=16, n_max=192, lanes=2, morton="ref63", tri_bend=True),
        # the differentiable workload: one 64x64 cloth, forward and backward with checkpoints
        dict(name="grad_64", kind="grad", n=64, steps=4, every=2),
        # the batched differentiable workload: cloths landing on icosphere meshes, some of them folded
        dict(name="grad_mesh_24", kind="grad_mesh", count=24, n_min=32, n_max=128, steps=2, every=2),
        # the LBVH microbenchmark: a million triangle boxes, 63-bit codes
        dict(name="lbvh_1m", kind="lbvh", count=1_000_000, morton="ref63"),
        # a small query: latency, 30-bit codes
        dict(name="lbvh_3k", kind="lbvh", count=3001, morton="k30"),
        # the caller-composed collision pipeline: LBVH pairs, continuous narrowphase, impulse response
        dict(name="pipeline_300", kind="pipeline", n=300, mode="ccd"),
        # the object-level broadphase, its default method, at the benchmark's size
        dict(name="objects_bvh_200k", kind="objects", method="bvh", count=200_000),
        # and a scene of some thousand objects on the spatial hash
        dict(name="objects_hash_20k", kind="objects", method="hash", count=20_011),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "drop", "batch", "host", "grad", "grad_mesh", "lbvh", "pipeline", "objects"])
    if kind == "step":
        fold = rng.random() < 0.6
        return dict(kind=kind, n=_log_int(rng, 16, 192), steps=1 if fold else rng.randint(1, 3), fold=fold,
                    wind=fold and rng.random() < 0.7, friction=fold and rng.random() < 0.3,
                    tri_bend=fold and rng.random() < 0.3, thickness=0.0)
    if kind == "drop":
        return dict(kind=kind, n=_log_int(rng, 160, 512))
    if kind in ("batch", "host"):
        return dict(kind=kind, count=_log_int(rng, 3, 110 if kind == "batch" else 40), n_min=rng.randint(16, 32),
                    n_max=rng.randint(60, 192), lanes=rng.choice([1, 2]), morton=rng.choice(["ref63", "ref63", "k30"]),
                    tri_bend=rng.random() < 0.25)
    if kind == "grad":
        return dict(kind=kind, n=rng.randint(20, 96), steps=rng.randint(2, 4), every=rng.randint(1, 4))
    if kind == "grad_mesh":
        return dict(kind=kind, count=_log_int(rng, 2, 32), n_min=rng.randint(24, 48), n_max=rng.randint(64, 128),
                    steps=rng.randint(1, 2), every=rng.randint(1, 2))
    if kind == "lbvh":
        return dict(kind=kind, count=_log_int(rng, 300, 1_000_000), morton=rng.choice(["ref63", "k30"]))
    if kind == "pipeline":
        return dict(kind=kind, n=_log_int(rng, 40, 300), mode=rng.choice(["ccd", "ccd", "dcd"]))
    return dict(kind=kind, method=rng.choice(["bvh", "bvh", "hash", "grid", "sap"]), count=_log_int(rng, 1000, 200_000))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _swing(spec, rng, fold: bool, calm: bool = False):
    """Positions and velocities of an n x n cloth (rest state: the flat grid
    of spec, pinned along z = 0) swinging about its pinned edge: rotated by an
    angle below the horizontal, pleated, moving at up to pendulum speed.
    fold: the part past a fold line lies back on the sheet, within about a
    thickness of it and closing, so that the layers are in contact.  calm: the
    first part of the swing, with shallow pleats."""
    n = spec.meta["n"]
    h = _thickness(spec)
    rest = spec.positions.astype(np.float64)
    u, w = rest[:, 0], rest[:, 2]
    th = rng.uniform(0.1, 0.35) if calm else rng.uniform(0.35, 1.25)
    tan = np.array([0.0, -math.sin(th), math.cos(th)])
    nrm = np.array([0.0, math.cos(th), math.sin(th)])
    s = w.copy()
    over = np.zeros_like(w)
    if fold:
        line = rng.uniform(0.75, 0.95)
        over = np.clip((w - line) * (n - 1) / 2.0, 0.0, 1.0)  # 0 on the sheet, 1 two rows past the fold
        s = np.where(w > line, 2.0 * line - w, w)
    waves, phase = rng.integers(1, 4), rng.uniform(0, 2 * math.pi)
    amp = rng.uniform(0.001, 0.004) if calm else rng.uniform(0.01, 0.05)
    ang = 2 * math.pi * waves * u + phase
    gap = h * (0.75 + 0.3 * np.sin(2 * math.pi * (2 * u + 3 * w)))
    off = amp * np.sin(ang) * s + over * gap
    pos = np.stack([rest[:, 0], np.full_like(u, 0.999), np.full_like(u, 0.001)], axis=1)
    pos = pos + s[:, None] * tan + off[:, None] * nrm + (rest - np.round(rest * (n - 1)) / (n - 1)) * 0.5
    omega = rng.uniform(0.4, 1.0) * math.sqrt(3.0 * 9.81 * math.sin(th))
    speed = -omega * s + 2.0 * amp * np.cos(ang) * s - over * rng.uniform(0.05, 0.3)
    vel = speed[:, None] * nrm + rng.normal(0.0, 0.003, size=pos.shape)
    pin = spec.pinned.astype(bool)
    pos[pin] = rest[pin]
    vel[pin] = 0.0
    pos[:, 1] = np.clip(pos[:, 1], 0.002, 0.999)
    return pos.astype(np.float32), vel.astype(np.float32)


def _landing(spec, rng, radius: float, fold: bool):
    """Positions and velocities of an unpinned cloth centred over a sphere at
    the origin, falling flat, its centre about to land; fold: a margin lies
    back on the sheet."""
    n = spec.meta["n"]
    h = _thickness(spec)
    pos = spec.positions.astype(np.float64)
    w = pos[:, 2] + 0.5
    over = np.zeros_like(w)
    z = pos[:, 2].copy()
    if fold:
        line = rng.uniform(0.85, 0.95)
        over = np.clip((w - line) * (n - 1) / 2.0, 0.0, 1.0)
        z = np.where(w > line, 2.0 * line - w - 0.5, z)
    speed = rng.uniform(1.5, 2.5)
    ang = 2 * math.pi * (rng.uniform(0.5, 1.5) * pos[:, 0] + rng.uniform(0.5, 1.5) * z)
    y = radius + h + rng.uniform(0.3, 0.6) * speed * DT + 0.003 * np.sin(ang) + over * h * (0.8 + 0.2 * np.sin(5 * ang))
    pos = np.stack([pos[:, 0], y + (pos[:, 1] - 1.0), z], axis=1)
    vel = np.stack([0.02 * np.cos(ang), -speed - over * 0.1, 0.02 * np.sin(ang)], axis=1)
    return pos.astype(np.float32), vel.astype(np.float32)


def _thickness(spec) -> float:
    p = spec.params
    return float(np.linalg.norm(spec.positions[0].astype(np.float64) - spec.positions[1]) / 3.0) \
        if p.thicknessFromMesh else p.thickness


def _stream():
    return torch.cuda.current_stream()


def _save(batch):
    n = C.c_uint64()
    _ffi.check(_ffi.lib().lc_batch_state_size(batch._h, C.byref(n)), "lc_batch_state_size")
    buf = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    _ffi.check(_ffi.lib().lc_batch_save_state(batch._h, C.c_void_p(buf.data_ptr()),
                                              C.c_void_p(_stream().cuda_stream)), "lc_batch_save_state")
    return buf


def _load(batch, buf) -> None:
    _ffi.check(_ffi.lib().lc_batch_load_state(batch._h, C.c_void_p(buf.data_ptr()),
                                              C.c_void_p(_stream().cuda_stream)), "lc_batch_load_state")


def _ready(batch, x, v):
    """The batch with the triangle order a rollout has at this state (one
    step from it), then put at the state itself."""
    put = lambda: batch.write_state(x.data_ptr(), x.data_ptr(), v.data_ptr(), False, _stream())  # noqa: E731
    put()
    batch.step(1, _stream())
    put()
    batch.sync()


def _outputs(batch, V: int):
    out = [torch.empty((V, 3), dtype=torch.float32, device="cuda") for _ in range(3)]
    batch.read_state(*(o.data_ptr() for o in out), False, _stream())
    return dict(x=out[0], x_prev=out[1], v=out[2])


def _step_spec(case: dict, seed: int):
    spec = scenes.small_cloth(seed=seed, n=case["n"])
    p = spec.params
    if case["thickness"] > 0.0:
        p.thickness = case["thickness"]
    else:
        p.thicknessFromMesh = 1
    if case["wind"]:
        rng = np.random.default_rng(seed + 5)
        scenes.set_constant_wind(p, (float(rng.uniform(-2, 2)), 0.0, float(rng.uniform(-2, 2))))
    p.useFriction = int(case["friction"])
    p.useTriangleBending = int(case["tri_bend"])
    return spec, *_swing(spec, np.random.default_rng(seed + 1), case["fold"])


def _drop_spec(case: dict, seed: int):
    spec = scenes.large_cloth(seed=seed, n=case["n"])
    return spec, *_landing(spec, np.random.default_rng(seed + 1), spec.params.sphereRadius, False)


def _sides(case: dict) -> np.ndarray:
    """The batch's cloth sides, the same for every seed: uniform over the
    range, largest first when the batch is cut into lanes by size."""
    sides = np.random.default_rng(case["count"]).integers(case["n_min"], case["n_max"] + 1, size=case["count"])
    return np.sort(sides)[::-1] if case.get("lanes", 1) > 1 else sides


def _batch_specs(case: dict, seed: int):
    """scenes.batched_cloths with the case's sides: stiffness U[0.5, 1],
    constant wind U[-2, 2] on x and z, two pinned corners.  A third of the
    cloths are folded."""
    specs, xs, vs = [], [], []
    for k, n in enumerate(int(q) for q in _sides(case)):
        rng = np.random.default_rng([seed, k])
        p = scenes.base_params(10, float(rng.uniform(0.5, 1.0)))
        p.dims[:] = (n, n)
        p.mortonMode = _ffi.LC_MORTON_K30 if case["morton"] == "k30" else _ffi.LC_MORTON_REF63
        p.useTriangleBending = int(case["tri_bend"])
        scenes.set_constant_wind(p, (float(rng.uniform(-2, 2)), 0.0, float(rng.uniform(-2, 2))))
        s = scenes.ClothSpec(scenes.grid_positions(n, rng), scenes.grid_indices(n), scenes.corner_pins(n), p,
                             dict(n=n))
        specs.append(s)
        x, v = _swing(s, rng, k % 3 == 0)
        xs.append(x)
        vs.append(v)
    return specs, np.concatenate(xs), np.concatenate(vs)


def _make_batch(case: dict, specs):
    lanes = min(case["lanes"], len(specs))
    return ClothBatchGroup(specs, lanes=lanes, order="given") if lanes > 1 else ClothBatch(specs)


def _mesh_specs(case: dict, seed: int):
    """scenes.batched_sphere_cloths with the case's sides: each cloth about
    to land on its own icosphere of subdivision 4, a third of them folded."""
    specs, xs, vs = [], [], []
    for k, n in enumerate(int(q) for q in _sides(case)):
        rng = np.random.default_rng([seed, k])
        r = float(rng.uniform(0.2, 0.4))
        s = scenes.icosphere_cloth(seed=seed + k, n=n, depth=4, radius=r, height=1.0)
        specs.append(s)
        x, v = _landing(s, rng, r, k % 3 == 0)
        xs.append(x)
        vs.append(v)
    return specs, np.concatenate(xs), np.concatenate(vs)


def _grad_spec(case: dict, seed: int):
    spec = scenes.adjoint_cloth(seed=seed, n=case["n"])
    return spec, *_swing(spec, np.random.default_rng(seed + 1), False, calm=True)


def _triangle_features(tri: np.ndarray) -> np.ndarray:
    """Ownership byte per triangle: the lowest triangle index owns a vertex
    (bits 5..3) or an edge (bits 2..0: v1v2, v2v3, v3v1)."""
    T = len(tri)
    f = np.zeros(3 * T, dtype=np.uint8)
    first = np.unique(tri.reshape(-1), return_index=True)[1]
    f[first] |= (1 << (5 - first % 3)).astype(np.uint8)
    t = tri.astype(np.int64)
    a, b = t, np.roll(t, -1, axis=1)
    key = (np.minimum(a, b) << 32 | np.maximum(a, b)).reshape(-1)
    first = np.unique(key, return_index=True)[1]
    f[first] |= (1 << (2 - first % 3)).astype(np.uint8)
    return np.bitwise_or.reduce(f.reshape(T, 3), axis=1)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    if kind in ("step", "drop", "batch"):
        if kind == "batch":
            specs, x, v = _batch_specs(case, seed)
            batch = _make_batch(case, specs)
        else:
            spec, x, v = _step_spec(case, seed) if kind == "step" else _drop_spec(case, seed)
            batch = ClothBatch([spec])
        _ready(batch, cuda(x), cuda(v))
        members = batch.batches if isinstance(batch, ClothBatchGroup) else [batch]
        return dict(case=case, batch=batch, start=[(m, _save(m)) for m in members], V=len(x))
    if kind == "host":
        specs, x, v = _batch_specs(case, seed)
        batch = _make_batch(case, specs)
        _ready(batch, cuda(x), cuda(v))
        pin = lambda a: torch.from_numpy(a).pin_memory()  # noqa: E731
        return dict(case=case, batch=batch, x=pin(x), v=pin(v),
                    out=[torch.empty(x.shape, dtype=torch.float32, pin_memory=True) for _ in range(3)])
    if kind in ("grad", "grad_mesh"):
        if kind == "grad":
            spec, x, v = _grad_spec(case, seed)
            specs = [spec]
        else:
            specs, x, v = _mesh_specs(case, seed)
        cloth = DiffCloth(specs, checkpoint_every=case["every"])
        xt, vt = cuda(x), cuda(v)
        _ready(cloth.batch, xt, vt)
        cloth.save(cloth.initial)
        rng = np.random.default_rng(seed + 2)
        ks, kb = (cuda(rng.uniform(0.6, 0.95, size=m).astype(np.float32)) for m in (cloth.E, cloth.B))
        g = cuda(rng.normal(size=x.shape).astype(np.float32))
        params = [t.requires_grad_(True) for t in (ks, kb, xt, vt)]
        return dict(case=case, cloth=cloth, params=params, g=g)
    if kind == "lbvh":
        lo, hi = scenes.random_triangle_boxes(case["count"], seed=seed)
        mode = _ffi.LC_MORTON_K30 if case["morton"] == "k30" else _ffi.LC_MORTON_REF63
        cap = max(1024, case["count"] // 2)
        return dict(case=case, lo=cuda(lo), hi=cuda(hi), tree=Lbvh(case["count"], 64, mode), cap=cap,
                    pairs=torch.zeros((cap, 2), dtype=torch.int32, device="cuda"))
    if kind == "pipeline":
        spec = scenes.small_cloth(seed=seed, n=case["n"])
        spec.params.thicknessFromMesh = 1
        xp, v = _swing(spec, np.random.default_rng(seed + 1), True)
        v = v * np.float32(0.2)  # slower than the swing: about ten pairs a triangle
        h = np.float32(_thickness(spec))
        x = xp + v * np.float32(DT)
        tri = spec.indices.astype(np.int64)
        both = np.stack([x[tri], xp[tri]], axis=1).reshape(len(tri), 6, 3)
        lo, hi = both.min(axis=1) - h, both.max(axis=1) + h
        T = len(tri)
        cap = 24 * T
        return dict(case=case, x=cuda(x), xp=cuda(xp), v=cuda(v), lo=cuda(lo), hi=cuda(hi),
                    tri=cuda(spec.indices.astype(np.int32)), feat=cuda(_triangle_features(spec.indices)),
                    fixed=cuda(spec.pinned), h=float(h), tree=Lbvh(T, 64),
                    narrow=Narrowphase(len(x), T, cap, 64 * T), cap=cap,
                    pairs=torch.zeros((cap, 2), dtype=torch.int32, device="cuda"),
                    contacts=[torch.zeros((4 * T, 12), dtype=torch.int32, device="cuda") for _ in range(2)])
    rng = np.random.default_rng(seed)
    lo = rng.uniform(0.0, 1.0, size=(case["count"], 3))
    hi = lo + rng.uniform(0.001, 0.01, size=lo.shape)
    return dict(case=case, lo=cuda(lo.astype(np.float32)), hi=cuda(hi.astype(np.float32)),
                pairs=torch.zeros((max(1024, case["count"]), 2), dtype=torch.int64, device="cuda"),
                bp=Broadphase(case["method"], case["count"], cell_size=0.02, table_size=1 << 18))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "drop", "batch"):
        for m, buf in state["start"]:
            _load(m, buf)
        state["batch"].step(case.get("steps", 1), _stream())
        return _outputs(state["batch"], state["V"])
    if kind == "host":
        x, v = state["x"].data_ptr(), state["v"].data_ptr()
        out = [o.data_ptr() for o in state["out"]]
        if isinstance(state["batch"], ClothBatchGroup):
            state["batch"].step_io(x, x, v, *out, True, _stream())
        else:
            state["batch"].write_state(x, x, v, True, _stream())
            state["batch"].step(1, _stream())
            state["batch"].read_state(*out, True, _stream())
        return dict(zip(("x", "x_prev", "v"), state["out"]))
    if kind in ("grad", "grad_mesh"):
        ks, kb, x, v = state["params"]
        out = ClothRollout.apply(state["cloth"], case["steps"], ks, kb, x, v)
        grads = torch.autograd.grad(out, state["params"], state["g"])
        return dict(x=out.detach(), **dict(zip(("k_stretch", "k_bend", "x0", "v0"), grads)))
    if kind == "lbvh":
        tree, n = state["tree"], case["count"]
        tree.build(state["lo"].data_ptr(), state["hi"].data_ptr(), n, _stream())
        k = tree.pairs(state["pairs"].data_ptr(), state["cap"], _stream())
        ids = torch.empty(n, dtype=torch.int32, device="cuda")
        tree.sorted_ids(ids.data_ptr(), _stream())
        return dict(count=k, pairs=state["pairs"], ids=ids)
    if kind == "pipeline":
        return _run_pipeline(state)
    state["bp"].update(state["lo"], state["hi"])
    pairs = state["bp"].test()
    state["pairs"][:len(pairs)] = pairs
    return dict(count=len(pairs), pairs=state["pairs"])


def _run_pipeline(state: dict):
    """LBVH pairs of the swept triangle boxes, the narrowphase on the
    triangles in the tree's order, and the impulse response on its contacts."""
    T, V = len(state["tri"]), len(state["x"])
    tree = state["tree"]
    tree.build(state["lo"].data_ptr(), state["hi"].data_ptr(), T, _stream())
    ids = torch.empty(T, dtype=torch.int32, device="cuda")
    tree.sorted_ids(ids.data_ptr(), _stream())
    k = min(tree.pairs(state["pairs"].data_ptr(), state["cap"], _stream()), state["cap"])
    order = ids.long()
    tri, feat = state["tri"][order].contiguous(), state["feat"][order].contiguous()
    mode = _ffi.LC_NARROW_CCD if state["case"]["mode"] == "ccd" else _ffi.LC_NARROW_DCD
    vf, ee = state["contacts"]
    rc, nvf, nee = state["narrow"].run(state["x"].data_ptr(), state["xp"].data_ptr(), state["v"].data_ptr(), V,
                                       tri.data_ptr(), feat.data_ptr(), T, state["pairs"].data_ptr(), k, state["h"],
                                       DT, vf.data_ptr(), len(vf), ee.data_ptr(), len(ee), _stream(), mode)
    _ffi.check(rc, "lc_narrowphase_run")
    x, v = state["x"].clone(), state["v"].clone()
    _ffi.check(_ffi.lib().lc_solve_collisions(
        C.c_void_p(x.data_ptr()), C.c_void_p(state["xp"].data_ptr()), C.c_void_p(v.data_ptr()),
        C.c_void_p(state["fixed"].data_ptr()), V, C.c_void_p(vf.data_ptr()), nvf, C.c_void_p(ee.data_ptr()), nee,
        0.9, 0.525 / V, DT, state["h"], C.c_void_p(_stream().cuda_stream)), "lc_solve_collisions")
    return dict(pairs=k, vf=nvf, ee=nee, vf_records=vf, ee_records=ee, x=x, v=v)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _mesh_counts(n: int):
    T = 2 * (n - 1) ** 2
    E = 2 * n * (n - 1) + (n - 1) ** 2
    return n * n, T, E, E - 4 * (n - 1)  # one bend for every inner edge


def _step_work(n: int, iters: int, steps: float = 1.0):
    """One cloth: the state read and written (x, x_prev, v, normals: 12 bytes
    each), topology, constraints and their parameters read; the solver's
    arithmetic (about 30 operations a stretch, 150 a bend) and about 200 per
    triangle for boxes, codes, sort and hierarchy."""
    V, T, E, B = _mesh_counts(n)
    return steps * (2 * 48 * V + 16 * T + 16 * E + 20 * B), steps * (iters * (30.0 * E + 150.0 * B) + 200.0 * T)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("step", "drop"):
        b, f = _step_work(case["n"], 20 if kind == "drop" else 10, case.get("steps", 1))
    elif kind in ("batch", "host"):
        b, f = np.sum([_step_work(int(n), 10) for n in _sides(case)], axis=0)
        if kind == "host":
            b += sum(5 * 12 * int(n) ** 2 for n in _sides(case))  # host to device (x, v) and back (3)
    elif kind in ("grad", "grad_mesh"):
        sides = [case["n"]] if kind == "grad" else _sides(case)
        # forward, the recorded re-run and the reverse pass of every step
        b, f = 3.0 * np.sum([_step_work(int(n), 10, case["steps"]) for n in sides], axis=0)
    elif kind == "lbvh":
        n = case["count"]
        pairs = min(64.0 * n, 0.065 * n * (n / 1e6))  # random boxes of 1e-3..5e-3 in the unit cube
        b, f = 24 * n + 4 * n + 8 * pairs, 200.0 * n
    elif kind == "pipeline":
        V, T, _, _ = _mesh_counts(case["n"])
        # boxes, triangles and state read, contacts (about one in four triangles) and state written
        b, f = 24 * T + 13 * T + 36 * V + 24 * V + 12 * T, 200.0 * T + 15 * 100.0 * T
    else:
        n = case["count"]
        b, f = 24 * n + 16 * (26_679 * (n / 200_000) ** 2), 200.0 * n
    return dict(bytes=float(b), flops=float(f))


# ---------------------------------------------------------------------------
# The contact-free step in 64 bits
# ---------------------------------------------------------------------------
class _Cloth64:
    """One cloth's constants: masses, edges with rest lengths, bends across
    the edges two triangles share, attachments to the pinned vertices."""

    def __init__(self, spec, device):
        t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=device)  # noqa: E731
        tri = spec.indices.astype(np.int64)
        rest = spec.positions.astype(np.float64)
        p = self.p = spec.params
        V = len(rest)
        a, b = tri.reshape(-1), np.roll(tri, -1, axis=1).reshape(-1)
        key = np.minimum(a, b) << 32 | np.maximum(a, b)
        order = np.argsort(key, kind="stable")
        new = np.ones(len(key), bool)
        new[1:] = key[order][1:] != key[order][:-1]
        first = np.sort(order[new])                       # edges in the order of their first triangle
        at = np.flatnonzero(~new)
        at = at[np.argsort(order[at], kind="stable")]     # bends in the order of the second
        t1, t2 = tri[order[at - 1] // 3], tri[order[at] // 3]
        shared = (t1[:, :, None] == t2[:, None, :]).any(axis=2)
        rows = np.arange(len(t1))
        last = 2 - np.argmax(shared[:, ::-1], axis=1)
        p1, p2 = t1[rows, last], t1[rows, np.argmax(shared, axis=1)]
        p3 = t1[rows, np.argmin(shared, axis=1)]
        p4 = t2[rows, np.argmax((t2 != p1[:, None]) & (t2 != p2[:, None]), axis=1)]
        self.s = t(np.stack([a[first], b[first]]), torch.int64)
        self.l0 = t(np.linalg.norm(rest[a[first]] - rest[b[first]], axis=1))
        self.b = t(np.stack([p1, p2, p3, p4]), torch.int64)
        pin = spec.pinned.astype(bool)
        vmass = float(p.objectMass) / V
        self.mass = t(np.where(pin, 1000.0, vmass))
        self.w = t(np.where(pin, 0.0, 1.0 / vmass))
        self.fixed = np.flatnonzero(pin)
        self.lra = [t(np.linalg.norm(rest - rest[f], axis=1) * (1.0 + p.strainLimit)) for f in self.fixed]
        cnt = np.bincount(np.concatenate([a[first], b[first], p1, p2, p3, p4]), minlength=V)
        self.count = t(cnt)
        self.h = _thickness(spec)
        self.g = t(np.array(list(p.gravity)))
        self.lo, self.hi = t(np.array(list(p.worldMin))), t(np.array(list(p.worldMax)))
        self.V = V

    def kp(self, k):
        return 1.0 - (1.0 - k) ** (1.0 / self.p.solverIterations)

    def bend(self, x, kp):
        p2, p3, p4 = (x[self.b[j]] for j in (1, 2, 3))
        w = [self.w[self.b[j]] for j in range(4)]
        c23, c24 = torch.linalg.cross(p2, p3), torch.linalg.cross(p2, p4)
        l23, l24 = c23.norm(dim=1), c24.norm(dim=1)
        ok = (l23 > 1e-8) & (l24 > 1e-8)
        n1, n2 = c23 / l23[:, None], c24 / l24[:, None]
        s, t = n1 + n2, n1 - n2
        ss, tt = (s * s).sum(1), (t * t).sum(1)
        ok = ok & (ss > 0)
        ss = torch.where(ok, ss, torch.ones_like(ss))
        gap = math.pi - float(np.float32(3.14159265359))
        term = torch.sqrt(0.25 * ss * tt) * (gap - 2.0 * torch.atan2(ss.sqrt(), tt.sqrt())) * kp
        u, v = s - n1 * (0.5 * ss)[:, None], s - n2 * (0.5 * ss)[:, None]
        q3 = torch.linalg.cross(p2, u) / l23[:, None]
        q4 = torch.linalg.cross(p2, v) / l24[:, None]
        q2 = -(torch.linalg.cross(p3, u) / l23[:, None] + torch.linalg.cross(p4, v) / l24[:, None])
        q = [-q2 - q3 - q4, q2, q3, q4]
        sf = sum(w[j] * (q[j] * q[j]).sum(1) for j in range(4))
        ok = ok & (sf > 1e-8)
        scale = torch.where(ok, term / torch.where(ok, sf, torch.ones_like(sf)), torch.zeros_like(term))
        return [q[j] * -(w[j] * scale)[:, None] for j in range(4)]

    def step(self, x, xp, v, kps, kpb):
        p, w, m = self.p, self.w, self.mass[:, None]
        dt = float(p.timestep)
        free = (w > 0)[:, None]
        v = (v + self.g * dt) * (1.0 - p.globalVelDamp)
        ms = self.mass.sum()
        xc, vc = (x * m).sum(0) / ms, (v * m).sum(0) / ms
        r = x - xc
        L = torch.linalg.cross(r, v * m).sum(0)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        inertia = (r * r * m).sum() * eye - (r * m).T @ r
        om = torch.linalg.solve(inertia, L)
        v = v + (vc + torch.linalg.cross(om.expand_as(r), r) - v) * p.kDamp
        x = xp + v * dt
        ground = float(p.worldMin[1]) + self.h
        on_ground = (x[:, 1] <= ground) if p.groundOn else torch.zeros_like(w, dtype=torch.bool)
        held = [((x - x[f]).norm(dim=1) > l0) & (w > 0) for f, l0 in zip(self.fixed, self.lra)]
        if p.sphereOn:
            x, xp = self.sphere(x, xp)
        for _ in range(p.solverIterations):
            acc = torch.zeros_like(x)
            cnt = self.count
            low = on_ground & (x[:, 1] < ground)
            acc = acc + torch.where(low, ground - x[:, 1], torch.zeros_like(w))[:, None] * eye[1]
            cnt = cnt + low
            for f, l0, on in zip(self.fixed, self.lra, held):
                d = torch.where(on[:, None], x - x[f], torch.ones_like(x))
                l = d.norm(dim=1, keepdim=True)
                acc = acc + torch.where(on[:, None], d / l * (l0[:, None] - l), torch.zeros_like(x))
                cnt = cnt + on
            d = x[self.s[0]] - x[self.s[1]]
            l = d.norm(dim=1, keepdim=True)
            w0, w1 = w[self.s[0]][:, None], w[self.s[1]][:, None]
            ws = w0 + w1
            tt = d / l * (l - self.l0[:, None]) * kps[:, None] / torch.where(ws > 0, ws, torch.ones_like(ws))
            acc = acc.index_add(0, self.s[0], -tt * w0).index_add(0, self.s[1], tt * w1)
            for j, c in enumerate(self.bend(x, kpb)):
                acc = acc.index_add(0, self.b[j], c)
            x = x + acc / cnt[:, None]
        v = torch.where(free, (x - xp) / dt, torch.zeros_like(x))
        xp = torch.where(free, x, xp)
        return torch.minimum(torch.maximum(x, self.lo), self.hi), xp, v

    def sphere(self, x, xp):
        c = torch.tensor(list(self.p.spherePos), dtype=x.dtype, device=x.device)
        rad = float(self.p.sphereRadius) + self.h
        d = x - xp
        l = d.norm(dim=1, keepdim=True)
        d = d / torch.where(l > 0, l, torch.ones_like(l))
        m = xp - c
        b, cc = (m * d).sum(1, keepdim=True), (m * m).sum(1, keepdim=True) - rad * rad
        disc = b * b - cc
        t = -b - disc.clamp(min=0).sqrt()
        hit = (l > 0) & ~((cc > 0) & (b > 0)) & (disc >= 0) & (t <= l)
        q = xp + d * t
        unit = lambda a: a / a.norm(dim=1, keepdim=True)  # noqa: E731
        on = c + unit(q - c) * rad
        inside = hit & (t < 0)
        xp = torch.where(inside, on + unit(on - c) * 1e-4, xp)
        x = torch.where(inside, on, torch.where(hit, q + unit(q - c) * 1e-4, x))
        return x, xp


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind not in ("step", "drop", "grad") or case.get("fold"):
        return None
    spec, x, v = {"step": _step_spec, "drop": _drop_spec, "grad": _grad_spec}[kind](case, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    cloth = _Cloth64(spec, device)
    x0, v0 = (torch.as_tensor(a, dtype=torch.float64, device=device) for a in (x, v))
    if kind != "grad":
        ones = torch.ones(1, dtype=torch.float64, device=device)
        kps, kpb = (cloth.kp(ones * float(k)) for k in (spec.params.kStretch, spec.params.kBend))
        s = (x0, x0, v0)
        with torch.no_grad():
            for _ in range(case.get("steps", 1)):
                s = cloth.step(*s, kps, kpb)
        return dict(zip(("x", "x_prev", "v"), s))
    rng = np.random.default_rng(seed + 2)
    params = [torch.as_tensor(rng.uniform(0.6, 0.95, size=m).astype(np.float32), dtype=torch.float64, device=device)
              for m in (cloth.s.shape[1], cloth.b.shape[1])] + [x0, v0]
    g = torch.as_tensor(rng.normal(size=x.shape).astype(np.float32), dtype=torch.float64, device=device)
    params = [t.requires_grad_(True) for t in params]
    ks, kb, x0, v0 = params
    s = (x0, x0, v0)
    for _ in range(case["steps"]):
        s = cloth.step(*s, cloth.kp(ks), cloth.kp(kb))
    grads = torch.autograd.grad(s[1], params, g)
    return dict(x=s[1].detach(), **dict(zip(("k_stretch", "k_bend", "x0", "v0"), grads)))
