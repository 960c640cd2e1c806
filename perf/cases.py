"""The work a user of this framework has it do, as cases that can be timed.

A case is a plain dict; ``prepare`` builds what a program holds before it
calls (scenes, device state, pinned result buffers), ``run`` is one pass
through the public API.  ``exact`` advances the same inputs in 64-bit torch
arithmetic written here from the method's formulas.

Kinds of pass:

* ``frame``     n substeps of one scene, then its positions (a render loop) or
                its whole particle records and bodies (an analysis loop)
* ``adaptive``  the stable timestep is estimated first and the frame is cut
                into that many substeps
* ``emitter``   a layer of particles enters, n substeps, the oldest leave
* ``job``       records from the host, n substeps, records back to the host
* ``batch``     n substeps of many independent scenes, then their positions
* ``served``    a burst of requests through the serving loop, to completion
"""
from __future__ import annotations

import math

import numpy as np
import torch

from slosh_b200 import scenes as S
from slosh_b200._lib import PARTICLE_DTYPE
from slosh_b200.batch import MpmBatch
from slosh_b200.pipeline import (
    GpuBoundaryCondition,
    MpmData,
    MpmPipeline,
    ParticleModel,
    RigidBody,
    SimulationParams,
    adaptive_substeps,
    make_particles,
)
from slosh_b200.serving import MpmServer

MATERIALS = ("fluid", "elastic", "sand")
# cell widths 1/k, powers of two and others; none puts a row of nodes exactly
# on the floor's surface (y = 0.05)
WIDTHS = (48, 56, 64, 72, 88, 96, 104, 112, 128)


def listed():
    return [
        # a small 3D scene stepped and drawn one substep at a time: latency
        {"name": "blob_3d_8k_single_step", "kind": "frame", "scene": "blob", "material": "fluid", "n": 8000, "k": 64,
         "substeps": 1, "full": False},
        # the 2D dam break of the configurations, ten substeps a frame
        {"name": "dam_break_2d_62k", "kind": "frame", "scene": "dam", "k": 256, "substeps": 10, "full": False},
        # the elastic drop of the configurations, its cubes tumbling, saved
        # whole every fifty substeps
        {"name": "elastic_drop_3d_524k", "kind": "frame", "scene": "drop", "k": 128, "substeps": 50, "full": True},
        # the headline sand column, twenty substeps a frame
        {"name": "sand_column_3d_4p7m", "kind": "frame", "scene": "column", "k": 256, "substeps": 20, "full": False,
         "two_way": False},
        # a mid-sized column with a cell width that is no power of two and a
        # cube the sand pushes; all records and bodies are read back
        {"name": "sand_two_way_3d_318k", "kind": "frame", "scene": "column", "k": 104, "substeps": 20, "full": True,
         "two_way": True},
        # several models and damping in one scene, round colliders
        {"name": "mixed_models_3d_61k", "kind": "frame", "scene": "mixed", "n": 61000, "k": 72, "substeps": 20,
         "full": True},
        # adaptive substepping of a 2D elastic sheet on round obstacles
        {"name": "adaptive_2d_25k", "kind": "adaptive", "material": "neo_hookean", "n": 25000, "k": 144,
         "frame_dt": 1.0e-3},
        # a faucet: particles are appended and removed every frame
        {"name": "emitter_3d_66k", "kind": "emitter", "n": 65536, "layer": 1024, "k": 64, "substeps": 20},
        # one whole job through host buffers
        {"name": "job_sand_3d_74k", "kind": "job", "material": "sand", "n": 74000, "k": 64, "substeps": 100},
        # the batched workload's scenes: mixed sizes, materials and widths
        {"name": "batch_mixed_48", "kind": "batch", "scenes": 48, "lo": 4000, "hi": 256000, "substeps": 20},
        # many small scenes of one size, as for sampling or learning
        {"name": "batch_small_64", "kind": "batch", "scenes": 64, "lo": 4000, "hi": 8000, "substeps": 10},
        # a burst of requests through the serving loop
        {"name": "served_12", "kind": "served", "requests": 12, "lo": 8000, "hi": 128000, "sub_lo": 50, "sub_hi": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("blob", "blob", "dam", "drop", "column", "mixed", "adaptive", "emitter", "job", "batch", "served"))
    substeps = rng.choice((1, 2, 5, 10, 20))
    if kind == "blob":
        return {"kind": "frame", "scene": "blob", "material": rng.choice(MATERIALS), "n": _log_int(rng, 6000, 2000000),
                "k": rng.choice(WIDTHS), "substeps": substeps, "full": rng.random() < 0.25}
    if kind == "dam":
        return {"kind": "frame", "scene": "dam", "k": rng.choice((64, 128, 256, 512)), "substeps": substeps, "full": False}
    if kind == "drop":
        return {"kind": "frame", "scene": "drop", "k": rng.choice((48, 64, 72, 96, 104, 128)), "substeps": substeps,
                "full": rng.random() < 0.25}
    if kind == "column":
        return {"kind": "frame", "scene": "column", "k": rng.choice((48, 64, 72, 96, 104, 128, 144, 192)),
                "substeps": substeps, "full": rng.random() < 0.25, "two_way": rng.random() < 0.5}
    if kind == "mixed":
        return {"kind": "frame", "scene": "mixed", "n": _log_int(rng, 9000, 600000), "k": rng.choice(WIDTHS),
                "substeps": substeps, "full": True}
    if kind == "adaptive":
        return {"kind": "adaptive", "material": rng.choice(("neo_hookean", "elastic", "sand")),
                "n": _log_int(rng, 4000, 400000), "k": rng.choice((96, 128, 144, 256)), "frame_dt": 1.0e-3}
    if kind == "emitter":
        return {"kind": "emitter", "n": _log_int(rng, 20000, 400000), "layer": rng.choice((256, 576, 1024)), "k": 64,
                "substeps": 20}
    if kind == "job":
        return {"kind": "job", "material": rng.choice(MATERIALS), "n": _log_int(rng, 8000, 400000),
                "k": rng.choice(WIDTHS), "substeps": rng.choice((10, 25, 50, 100))}
    if kind == "batch":
        lo = _log_int(rng, 4000, 20000)
        return {"kind": "batch", "scenes": rng.randrange(4, 65), "lo": lo, "hi": lo + _log_int(rng, 1000, 100000),
                "substeps": rng.choice((5, 10, 20))}
    return {"kind": "served", "requests": rng.randrange(3, 13), "lo": 8000, "hi": _log_int(rng, 20000, 128000),
            "sub_lo": 30, "sub_hi": rng.randrange(60, 200)}


# -- scenes -------------------------------------------------------------------


def _floor(k):
    t = 4.0 / k
    return RigidBody(("cuboid", (4.0, t, 4.0)), translation=(0.5, 0.05 - t, 0.5))


def _tumble(parts, seed):
    """Turns a body of particles about its centre, so that it strains from
    the first substep on."""
    x = parts["position"].astype(np.float64)
    w = np.random.default_rng(seed + 11).normal(0.0, 2.0, 3)
    parts["velocity"] = np.cross(w, x - x.mean(0))


def _mixed_scene(n, k, seed):
    """Three blobs side by side: fixed-corotated, Neo-Hookean with damping
    and Neo-Hookean sand, over a floor with a ball and a capsule."""
    rng = np.random.default_rng(seed)
    h = 1.0 / k
    side = max((n / 24.0) ** (1.0 / 3.0) * h, 4 * h)
    models = (
        (ParticleModel.elastic(1.0e5, 0.3), 1000.0, 0.0),
        (ParticleModel.elastic_neo_hookean(8.0e4, 0.25), 900.0, 0.5),
        (ParticleModel.sand_neo_hookean(3.0e5, 0.3, friction_angle_deg=32.0), 2000.0, 0.0),
    )
    parts = []
    for i, (model, density, damping) in enumerate(models):
        lo = np.array([0.5 + (i - 1.5) * (side + 2 * h), 0.1, 0.5 - side / 2])
        pts = S._jitter(S._lattice(tuple(lo), tuple(lo + side), h / 2), h / 4, rng)
        p = make_particles(pts, h / 4, density, model, dim=3)
        p["velocity"][:, :3] = rng.normal(0.0, 0.2, 3)
        p["damping"] = damping
        parts.append(p)
    bodies = [
        _floor(k),
        RigidBody(("ball", 0.06), translation=(0.5 - side, 0.11 - h * 0.3, 0.5), boundary_condition=GpuBoundaryCondition.slip()),
        RigidBody(("capsule", ((-0.2, 0.0, 0.0), (0.2, 0.0, 0.0), 0.03)), translation=(0.5, 0.1, 0.5),
                  boundary_condition=GpuBoundaryCondition.stick()),
    ]
    parts = np.concatenate(parts)
    return S.Scene("mixed", 3, h, SimulationParams((0.0, -9.81, 0.0), 5.0e-5), parts, bodies, 100,
                   S._grid_capacity(len(parts), 8, 3))


def _sheet_2d(case, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / case["k"]
    side = math.sqrt(case["n"] / 4.0) * h
    pts = S._jitter(S._lattice((0.5 - side / 2, 0.3), (0.5 + side / 2, 0.3 + side), h / 2), h / 4, rng)
    model = {"neo_hookean": ParticleModel.elastic_neo_hookean(1.0e5, 0.3), "elastic": ParticleModel.elastic(1.0e5, 0.3),
             "sand": ParticleModel.sand(1.0e5, 0.3, friction_angle_deg=30.0)}[case["material"]]
    parts = make_particles(pts, h / 4, 1000.0, model, dim=2)
    parts["velocity"][:, 1] = -1.0 - rng.random()
    t = 4.0 * h
    bodies = [
        RigidBody(("cuboid", (8.0, t)), translation=(0.5, 0.05 - t), rotation=0.0),
        RigidBody(("ball", 0.08), translation=(0.4, 0.235), rotation=0.0, boundary_condition=GpuBoundaryCondition.slip()),
        RigidBody(("capsule", ((-0.1, 0.0), (0.1, 0.0), 0.03)), translation=(0.62, 0.28), rotation=0.3,
                  boundary_condition=GpuBoundaryCondition.stick()),
    ]
    return S.Scene("sheet_2d", 2, h, SimulationParams((0.0, -9.81), 1.0e-4), parts, bodies, 100,
                   S._grid_capacity(len(parts), 4, 2))


def _emitter(case, seed):
    """A pool on the floor and one layer (a square of `layer` particles)
    that enters 0.2 above it at 4 m/s."""
    k, h = case["k"], 1.0 / case["k"]
    pool = S.random_scene_3d(case["n"], "fluid", h, seed)
    rng = np.random.default_rng(seed + 1)
    m = int(round(math.sqrt(case["layer"])))
    xs = 0.5 + (np.arange(m) + 0.5 - m / 2) * h / 2
    top = float(pool.particles["position"][:, 1].max()) + 0.2
    pts = np.array([(x, top, z) for x in xs for z in xs])
    pts = S._jitter(pts, h / 4, rng)
    layer = make_particles(pts, h / 4, 1000.0, ParticleModel.fluid_tait(1000.0, 1.0e4, 7.0), dim=3)
    layer["velocity"][:, 1] = -4.0
    return pool, layer


def _scene(case, seed):
    kind = case.get("scene", case["kind"])
    if kind == "dam":
        return S.dam_break_2d(h=1.0 / case["k"], seed=seed)
    if kind == "drop":
        sc = S.elastic_drop_3d(h=1.0 / case["k"], seed=seed)
        half = sc.n // 2
        _tumble(sc.particles[:half], seed)
        _tumble(sc.particles[half:], seed + 1)
        return sc
    if kind == "column":
        return S.sand_column_3d(h=1.0 / case["k"], seed=seed, cube_coupling="two_way" if case["two_way"] else "one_way")
    if kind == "mixed":
        return _mixed_scene(case["n"], case["k"], seed)
    if kind == "adaptive":
        return _sheet_2d(case, seed)
    sc = S.random_scene_3d(case["n"], case["material"], 1.0 / case["k"], seed)  # blob, job
    _tumble(sc.particles, seed)
    return sc


def _scene_list(case, seed, count):
    rng = np.random.default_rng(case["lo"] + case["hi"])  # the mix is the case's, the particles are the seed's
    ns = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), count))
    mats = rng.choice(MATERIALS, count)
    ks = rng.choice((64, 128), count)
    return [S.random_scene_3d(int(n), str(m), 1.0 / int(k), seed=seed * 1000 + i)
            for i, (n, m, k) in enumerate(zip(ns, mats, ks))]


# -- what a program holds -------------------------------------------------------


def _pinned(n, dtype, cols=None):
    dt = np.dtype(dtype)
    buf = torch.empty(max(n * dt.itemsize * (cols or 1), 1), dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    a = buf.numpy()[: n * dt.itemsize * (cols or 1)].view(dt)
    a[...] = np.zeros((), dt)
    return a.reshape(n, cols) if cols else a


def _data(scene, extra=0):
    # room for the scene to spread out: four times the blocks it starts with
    return MpmData(scene.params, scene.particles, scene.bodies, cell_width=scene.cell_width,
                   grid_capacity=max(scene.grid_capacity, 16384), dim=scene.dim, max_particles=scene.n + extra)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind, "pipe": MpmPipeline()}
    if kind in ("frame", "adaptive"):
        sc = _scene(case, seed)
        st["data"] = _data(sc)
        st["params"] = sc.params
        if kind == "adaptive" or case["full"]:
            st["out"] = _pinned(sc.n, PARTICLE_DTYPE)
        else:
            st["out"] = _pinned(sc.n, np.float32, 4)
    elif kind == "emitter":
        pool, layer = _emitter(case, seed)
        st["data"] = _data(pool, extra=len(layer))
        st["layer"] = layer
        st["out"] = _pinned(pool.n, np.float32, 4)
    elif kind == "job":
        sc = _scene(case, seed)
        st["data"] = _data(sc)
        st["host"] = _pinned(sc.n, PARTICLE_DTYPE)
        st["host"][:] = sc.particles
        st["out"] = _pinned(sc.n, PARTICLE_DTYPE)
    elif kind == "batch":
        scs = _scene_list(case, seed, case["scenes"])
        total = sum(sc.n for sc in scs)
        blocks = int(sum(max(1024, 5.0 * sc.n / 512.0) for sc in scs))
        b = MpmBatch(3, max_particles=total, grid_capacity=blocks, max_scenes=len(scs), max_bodies=2 * len(scs))
        st["batch"] = b
        st["out"] = _pinned(total, np.float32, 4)
        st["slots"], at = [], 0
        for sc in scs:
            st["slots"].append((b.add(sc), st["out"][at : at + sc.n]))
            at += sc.n
    else:
        rng = np.random.default_rng(case["sub_lo"] + case["sub_hi"])
        st["requests"] = [(sc, int(rng.integers(case["sub_lo"], case["sub_hi"] + 1)))
                          for sc in _scene_list(case, seed, case["requests"])]
        st["server"] = MpmServer(4 << 30, max_scenes=64, max_bodies=256)
    return st


def _records(out):
    return {"position": out["position"], "velocity": out["velocity"], "def_grad": out["def_grad"],
            "affine": out["affine"], "plastic": out["model"][:, :3], "enabled": out["enabled"]}


def run(st):
    case, kind, pipe = st["case"], st["kind"], st["pipe"]
    if kind == "frame":
        data = st["data"]
        pipe.launch_step(data, case["substeps"])
        if not case["full"]:
            return {"positions": data.positions(st["out"])}
        res = _records(data.download_particles(st["out"]))
        bodies = data.get_bodies()
        res["translation"], res["linvel"] = bodies["translation"], bodies["linvel"]
        return res
    if kind == "adaptive":
        data = st["data"]
        bound = pipe.compute_timestep_bound(data)
        n = adaptive_substeps(case["frame_dt"], bound, 1, 40)
        data.set_params(SimulationParams(st["params"].gravity, case["frame_dt"] / n))
        pipe.launch_step(data, n)
        res = _records(data.download_particles(st["out"]))
        res["bound"] = bound
        return res
    if kind == "emitter":
        data = st["data"]
        data.append(st["layer"])
        pipe.launch_step(data, case["substeps"])
        data.shift_remove(0, len(st["layer"]))
        return {"positions": data.positions(st["out"])}
    if kind == "job":
        data = st["data"]
        data.upload(st["host"])
        pipe.launch_step(data, case["substeps"])
        return _records(data.download_particles(st["out"]))
    if kind == "batch":
        b = st["batch"]
        b.step(case["substeps"])
        for slot, out in st["slots"]:
            b.positions(slot, out)
        return {"positions": st["out"]}
    srv = st["server"]
    rids = [srv.submit(sc.particles, sc.cell_width, sc.params, sc.bodies, sub)[0] for sc, sub in st["requests"]]
    got = {}
    while len(got) < len(rids):
        srv.wait_idle()
        for c in srv.poll():
            if c["status"] != 0:
                raise RuntimeError("request failed with status %d" % c["status"])
            got[c["id"]] = c["positions"]
    return [got[r] for r in rids]


# -- what a pass cannot do without ----------------------------------------------

# Per particle and substep: x, v, C and F (a fluid: its volume ratio) read and
# written, mass, volume and material read, three words of plastic state read
# and written for sand.  FLOPs from the method's sums over the stencil (P2G
# about 0.7 k, G2P 0.8 k in 3D; a third of that in 2D) and the model.
_FLOPS = {"fluid": 100, "elastic": 600, "neo_hookean": 150, "sand": 800, "mixed": 550}


def _per_particle(dim, material):
    mat = dim * dim
    state = 2 * dim + mat + (1 if material == "fluid" else mat)
    words = 2 * state + 3 + (6 if material in ("sand", "mixed") else 0)
    return 4.0 * words, (1500.0 if dim == 3 else 450.0) + _FLOPS[material]


def _blob_n(n, k):
    side = max((n / 8.0) ** (1.0 / 3.0), 4.0)
    return float(math.floor(2 * side + 1e-9)) ** 3


def work(case):
    kind, sub = case["kind"], case.get("substeps", 1)
    dim, extra = 3, 0.0
    if kind in ("frame", "job"):
        scene = case.get("scene", "blob")
        k = case["k"]
        if scene == "dam":
            dim, mat, n = 2, "fluid", math.floor(0.8 * k + 1e-9) * math.floor(1.2 * k + 1e-9)
        elif scene == "drop":
            mat, n = "elastic", 2.0 * math.floor(0.5 * k + 1e-9) ** 3
        elif scene == "column":
            mat, n = "sand", math.pi * 0.15**2 * 0.5 * 8.0 * k**3
        elif scene == "mixed":
            mat, n = "mixed", case["n"]
        else:
            mat, n = case["material"], _blob_n(case["n"], k)
        extra = n * (192.0 if case.get("full", kind == "job") else 16.0) + (n * 192.0 if kind == "job" else 0.0)
    elif kind == "adaptive":
        dim, mat, n = 2, case["material"], case["n"]
        sub = 5
        extra = n * 192.0 + n * 24.0
    elif kind == "emitter":
        mat, n = "fluid", case["n"] + case["layer"]
        extra = case["n"] * 16.0 + case["layer"] * 192.0
    elif kind == "batch":
        mat = "elastic"
        n = case["scenes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        extra = n * 16.0
    else:
        mat = "elastic"
        n = case["requests"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        sub = 0.5 * (case["sub_lo"] + case["sub_hi"])
        extra = n * (16.0 + 192.0)
    b, f = _per_particle(dim, mat)
    return {"bytes": n * sub * b + extra, "flops": n * sub * f}


# -- the method in 64 bits ------------------------------------------------------


def _f32(v):
    return float(np.float32(v))


def _eig_sym(b, sweeps=5):
    """Eigenvalues and eigenvectors of symmetric (n, d, d) matrices by cyclic
    Jacobi rotations; d = 2 or 3."""
    d = b.shape[-1]
    a = [[b[:, i, j].clone() for j in range(d)] for i in range(d)]
    one, zero = torch.ones_like(a[0][0]), torch.zeros_like(a[0][0])
    V = [[one.clone() if i == j else zero.clone() for j in range(d)] for i in range(d)]
    for _ in range(sweeps):
        for p in range(d):
            for q in range(p + 1, d):
                apq = a[p][q]
                nz = apq != 0
                theta = (a[q][q] - a[p][p]) / (2.0 * torch.where(nz, apq, one))
                t = torch.where(theta >= 0, one, -one) / (theta.abs() + torch.sqrt(theta * theta + 1.0))
                t = torch.where(nz, t, zero)
                c = torch.rsqrt(t * t + 1.0)
                s = t * c
                a[p][p], a[q][q] = a[p][p] - t * apq, a[q][q] + t * apq
                a[p][q] = a[q][p] = zero
                for r in range(d):
                    if r != p and r != q:
                        x, y = a[r][p], a[r][q]
                        a[r][p] = a[p][r] = c * x - s * y
                        a[r][q] = a[q][r] = s * x + c * y
                    x, y = V[r][p], V[r][q]
                    V[r][p], V[r][q] = c * x - s * y, s * x + c * y
    lam = torch.stack([a[i][i] for i in range(d)], 1)
    return lam, torch.stack([torch.stack(row, 1) for row in V], 1)


def _det(F):
    if F.shape[-1] == 2:
        return F[:, 0, 0] * F[:, 1, 1] - F[:, 0, 1] * F[:, 1, 0]
    return (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1)


class _Exact:
    """The scene's particles and bodies in float64."""

    def __init__(self, parts, bodies, h, params, dim):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.dim, self.h = dim, _f32(h)
        self.gravity = [_f32(g) for g in list(params.gravity)[:dim]]
        self.dt = _f32(params.dt)
        self.bodies = [self._body(b) for b in bodies]
        self.dynamic = any(b["two_way"] for b in self.bodies)
        self.load(parts)

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a).astype(np.float64)).to(self.dev)

    def load(self, parts):
        d, n = self.dim, len(parts)
        self.x, self.v = self.t(parts["position"][:, :d]), self.t(parts["velocity"][:, :d])
        self.F = self.t(parts["def_grad"].reshape(n, 3, 3).transpose(0, 2, 1)[:, :d, :d])
        self.C = self.t(parts["affine"].reshape(n, 3, 3).transpose(0, 2, 1)[:, :d, :d])
        self.m, self.V0 = self.t(parts["mass"]), self.t(parts["init_volume"])
        self.damp = self.t(parts["damping"])
        self.model = self.t(parts["model"])
        self.tags = parts["model_tag"].copy()
        self.sets = [(int(t), torch.from_numpy(np.flatnonzero(self.tags == t)).to(self.dev)) for t in np.unique(self.tags)]

    def append(self, parts):
        other = _Exact.__new__(_Exact)
        other.dim, other.dev = self.dim, self.dev
        other.load(parts)
        for k in ("x", "v", "F", "C", "m", "V0", "damp", "model"):
            setattr(self, k, torch.cat([getattr(self, k), getattr(other, k)]))
        self.tags = np.concatenate([self.tags, other.tags])
        self.sets = [(int(t), torch.from_numpy(np.flatnonzero(self.tags == t)).to(self.dev)) for t in np.unique(self.tags)]

    def _body(self, b):
        r = b.record(self.dim)
        d = self.dim
        out = {"kind": b.shape[0], "a": r["shape_a"].astype(np.float64), "b": r["shape_b"].astype(np.float64),
               "rot": r["rotation"].astype(np.float64), "tra": r["translation"][:d].astype(np.float64),
               "scale": float(r["translation"][3]), "lin": r["linvel"][:3].astype(np.float64),
               "ang": r["angvel"][:3].astype(np.float64), "inv_mass": r["inv_mass"][:d].astype(np.float64),
               "bc": int(r["bc_type"]), "friction": float(r["bc_friction"]), "two_way": int(r["coupling"]) == 1}
        if d == 3:
            R = _rotation(out["rot"], 3)
            out["inertia"] = R.T @ r["inv_inertia"].astype(np.float64).reshape(3, 4)[:, :3].T @ R
        else:
            out["inertia"] = float(r["inv_inertia"][0])
        return out

    # closest boundary point of a body for the points P, and whether inside
    def _project(self, b, P):
        d = self.dim
        R = self.t(_rotation(b["rot"], d))
        tra = self.t(b["tra"])
        L = (P - tra) @ R / b["scale"]
        if b["kind"] == "cuboid":
            he = self.t(b["a"][:d])
            clamped = torch.minimum(torch.maximum(L, -he), he)
            inside = (L == clamped).all(1)
            sg = torch.where(L > 0, 1.0, -1.0).double()
            diff = he - sg * L
            axis = diff.argmin(1, keepdim=True)
            inner = L.scatter(1, axis, (L + diff * sg).gather(1, axis))
            Q = torch.where(inside[:, None], inner, clamped)
        elif b["kind"] == "ball":
            dist = L.norm(dim=1)
            Q = L * (b["a"][0] / torch.where(dist > 0, dist, torch.ones_like(dist)))[:, None]
            inside = dist <= b["a"][0]
        else:  # capsule
            a0, ab = self.t(b["a"][:d]), self.t(b["b"][:d] - b["a"][:d])
            u = ((L - a0) @ ab / (ab @ ab)).clamp(0.0, 1.0)
            q = a0 + u[:, None] * ab
            dv = L - q
            dist = dv.norm(dim=1)
            Q = q + dv * (b["b"][3] / torch.where(dist > 0, dist, torch.ones_like(dist)))[:, None]
            inside = dist <= b["b"][3]
        return Q * b["scale"] @ R.T + tra, inside

    def _collide(self, P):
        """Collider id (-1: none), normal and signed distance of the points."""
        n = len(P)
        cap = 1.5 * self.h
        best = torch.full((n,), 1.0e10, dtype=torch.float64, device=self.dev)
        cid = torch.full((n,), -1, dtype=torch.int64, device=self.dev)
        N, B = torch.zeros_like(P), torch.zeros_like(P)
        for i, b in enumerate(self.bodies):
            Q, inside = self._project(b, P)
            dp = Q - P
            dist = dp.norm(dim=1)
            sign = torch.where(inside, -1.0, 1.0).double()
            take = (inside | (dp.abs() <= cap).all(1)) & (sign * dist < best) & (dist != 0)
            nn = dp / (torch.where(dist != 0, dist, torch.ones_like(dist)) * -sign)[:, None]
            N = torch.where(take[:, None], nn, N)
            B = torch.where(take[:, None], Q, B)
            cid = torch.where(take, i, cid)
            best = torch.where(take, dist, best)
        return cid, N, ((P - B) * N).sum(1)

    def _boundary(self, bc, friction, vel, n, dist):
        near = (dist <= 0)[:, None]
        nv = (vel * n).sum(1, keepdim=True)
        if bc == 0:
            return torch.where(near, torch.zeros_like(vel), vel)
        if bc == 1:
            return torch.where(near, vel - n * nv, vel)
        if bc in (2, 3):
            tv = vel - n * nv
            tl = tv.norm(dim=1, keepdim=True)
            sc = (tl + friction * nv).clamp(min=0.0)
            hit = torch.where(tl > 1.0e-8, tv / torch.where(tl > 0, tl, torch.ones_like(tl)), torch.zeros_like(tv)) * sc
            soon = torch.where(-nv * self.dt > dist[:, None], vel - (dist[:, None] / self.dt + nv) * n, vel)
            return torch.where(nv < 0, torch.where(near, hit, soon), vel)
        return vel

    def step(self):
        d, h, dt = self.dim, self.h, self.dt
        x = self.x
        base = torch.round(x / h).to(torch.int64) - 1
        lo = base.min(0).values
        dims = [int(v) + 4 for v in (base.max(0).values - lo)]
        strides = [1]
        for q in dims[:-1]:
            strides.append(strides[-1] * q)
        total = strides[-1] * dims[-1]
        cell = sum((base[:, i] - lo[i]) * strides[i] for i in range(d))
        d0 = base.double() * h - x
        f = -d0 / h
        w = torch.stack([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1.0) ** 2, 0.5 * (f - 0.5) ** 2], 2)
        offs = [(i, j, k) for k in range(3 if d == 3 else 1) for j in range(3) for i in range(3)]
        grid = torch.zeros(total, d + 1, dtype=torch.float64, device=self.dev)
        mom = self.v * self.m[:, None] + torch.einsum("nij,nj->ni", self.C, d0)
        for o in offs:
            wt = w[:, 0, o[0]] * w[:, 1, o[1]]
            if d == 3:
                wt = wt * w[:, 2, o[2]]
            shift = torch.tensor(o[:d], dtype=torch.float64, device=self.dev) * h
            val = torch.cat([mom + self.C @ shift, self.m[:, None]], 1) * wt[:, None]
            grid.index_add_(0, cell + sum(o[i] * strides[i] for i in range(d)), val)
        # grid update on the nodes with mass
        node = torch.nonzero(grid[:, d] > 0).squeeze(1)
        mass = grid[node, d]
        g = torch.tensor(self.gravity, dtype=torch.float64, device=self.dev)
        vel = ((grid[node, :d] + mass[:, None] * g * dt) / mass[:, None]).clamp(-h / dt, h / dt)
        P = torch.stack([(node // strides[i] % dims[i] + lo[i]).double() * h for i in range(d)], 1)
        cid, N, sd = self._collide(P)
        push = []
        for i, b in enumerate(self.bodies):
            s = torch.nonzero(cid == i).squeeze(1)
            if not b["two_way"]:
                vel[s] = self._boundary(b["bc"], b["friction"], vel[s], N[s], sd[s] - h)
                continue
            r = P[s] - self.t(b["tra"])
            if d == 3:
                vb = self.t(b["lin"]) + torch.linalg.cross(self.t(b["ang"]).expand_as(r), r)
            else:
                vb = self.t(b["lin"][:2]) + b["ang"][0] * torch.stack([-r[:, 1], r[:, 0]], 1)
            new = self._boundary(b["bc"], b["friction"], vel[s] - vb, N[s], sd[s] - h) + vb
            J = mass[s, None] * (vel[s] - new)
            vel[s] = new
            torque = torch.linalg.cross(r, J).sum(0) if d == 3 else (r[:, 0] * J[:, 1] - r[:, 1] * J[:, 0]).sum()
            push.append((b, J.sum(0).cpu().numpy(), torque.cpu().numpy()))
        grid[:, :d] = 0.0
        grid[node, :d] = vel
        # gather
        v = torch.zeros_like(self.v)
        grad = torch.zeros_like(self.C)
        for o in offs:
            wt = w[:, 0, o[0]] * w[:, 1, o[1]]
            if d == 3:
                wt = wt * w[:, 2, o[2]]
            gv = grid[cell + sum(o[i] * strides[i] for i in range(d)), :d] * wt[:, None]
            v += gv
            grad += gv[:, :, None] * (d0 + torch.tensor(o[:d], dtype=torch.float64, device=self.dev) * h)[:, None, :]
        inv_d = 4.0 / (h * h)
        grad *= inv_d
        speed = v.norm(dim=1, keepdim=True)
        v = torch.where(speed > h / dt, v / torch.where(speed > 0, speed, torch.ones_like(speed)) * h / dt, v)
        v = v / (1.0 + self.damp * dt)[:, None]
        self.v, self.x = v, x + v * dt
        tau = torch.zeros_like(grad)
        for tag, s in self.sets:
            tau[s] = self._model(tag, s, grad[s])
        self.C = grad * self.m[:, None, None] - tau * (self.V0 * inv_d * dt)[:, None, None]
        self._move_bodies(push)

    def _model(self, tag, s, grad):
        d, dt = self.dim, self.dt
        eye = torch.eye(d, dtype=torch.float64, device=self.dev)
        p = self.model[s]
        if tag == 4:  # Tait fluid: the volume ratio is F00
            J = self.F[s, 0, 0]
            J = J + J * grad.diagonal(dim1=1, dim2=2).sum(1) * dt
            self.F[s] = J[:, None, None] * eye
            pressure = p[:, 1] / p[:, 2] * (J ** -p[:, 2] - 1.0)
            return (-J * pressure)[:, None, None] * eye
        F = self.F[s]
        F = F + dt * grad @ F
        lam, mu = (p[:, 0], p[:, 1]) if tag in (0, 1) else (p[:, 9], p[:, 10])
        U = sv = None
        if tag != 1:
            e, U = _eig_sym(F @ F.transpose(1, 2))
            sv = torch.sqrt(e)
        if tag in (2, 3):
            F, sv = self._drucker_prager(s, p, F, U, sv)
        self.F[s] = F
        if tag in (1, 3):
            J = _det(F).clamp(min=1.0e-10)
            return mu[:, None, None] * (F @ F.transpose(1, 2)) + (lam * torch.log(J) - mu)[:, None, None] * eye
        J = sv.prod(1)
        diag = 2.0 * mu[:, None] * (sv - 1.0) * sv + (lam * (J - 1.0) * J)[:, None]
        return (U * diag[:, None, :]) @ U.transpose(1, 2)

    def _drucker_prager(self, s, p, F, U, sv):
        d = float(self.dim)
        q, vol = p[:, 1], p[:, 2]
        lam, mu = p[:, 7], p[:, 8]
        angle = p[:, 3] + (p[:, 4] * q - p[:, 6]) * torch.exp(-p[:, 5] * q)
        sa = torch.sin(angle)
        alpha = math.sqrt(2.0 / 3.0) * 2.0 * sa / (3.0 - sa)
        ls = torch.log(sv)
        strain = ls + vol[:, None] / d
        tr = strain.sum(1)
        dev = strain - tr[:, None] / d
        tip = (tr > 0) | (dev == 0).all(1)
        devn = dev.norm(dim=1)
        gamma = devn + (d * lam + 2.0 * mu) / (2.0 * mu) * tr * alpha
        hh = strain - dev * (gamma / torch.where(devn > 0, devn, torch.ones_like(devn)))[:, None]
        hh = torch.where(tip[:, None], torch.zeros_like(hh), hh)
        dq = torch.where(tip, strain.norm(dim=1), gamma)
        go = tip | (gamma > 0)
        ns = torch.where(go[:, None], torch.exp(hh), sv)
        new = p.clone()
        new[:, 0] = torch.where(go, p[:, 0] * sv.prod(1) / ns.prod(1), p[:, 0])
        new[:, 1] = torch.where(go, q + dq, q)
        new[:, 2] = torch.where(go, vol + ls.sum(1) - hh.sum(1), vol)
        self.model[s] = new
        M = (U * (ns / sv)[:, None, :]) @ U.transpose(1, 2)
        return torch.where(go[:, None, None], M @ F, F), ns

    def _move_bodies(self, push):
        d, dt = self.dim, self.dt
        for b, J, A in push:
            b["lin"][:d] += b["inv_mass"] * J
            if d == 3:
                R = _rotation(b["rot"], 3)
                b["ang"] += R @ b["inertia"] @ R.T @ A
            else:
                b["ang"][0] += b["inertia"] * float(A)
            ln, an = np.linalg.norm(b["lin"][:d]), np.linalg.norm(b["ang"][: 3 if d == 3 else 1])
            if np.any(J != 0) or np.any(A != 0):
                if ln > 0.1 * self.h / dt:
                    b["lin"][:d] *= 0.1 * self.h / dt / ln
                if an > 1.0:
                    b["ang"] *= 1.0 / an
        for b in self.bodies:
            if d == 3:
                b["rot"] = _spin(b["rot"], b["ang"] * dt)
            else:
                c, sn = math.cos(b["ang"][0] * dt), math.sin(b["ang"][0] * dt)
                b["rot"][:2] = c * b["rot"][0] - sn * b["rot"][1], sn * b["rot"][0] + c * b["rot"][1]
            b["tra"] = b["tra"] + b["lin"][:d] * dt
            b["lin"][:d] += np.asarray(self.gravity) * (b["inv_mass"] != 0) * dt

    def timestep_bound(self):
        """The smallest of each particle's sound-speed and velocity bounds, in
        whole picoseconds (elastic and sand models)."""
        J = _det(self.F)
        vlen = self.v.norm(dim=1)
        best = math.inf
        for tag, s in self.sets:
            lam, mu, cfl = (self.model[s, i + (0 if tag in (0, 1) else 9)] for i in range(3))
            rho = self.m[s] / self.V0[s] / J[s].clamp(min=1.0e-6)
            c = torch.sqrt((lam + 2.0 * mu / 3.0 + 4.0 * mu / 3.0) / rho)
            dt = torch.minimum(cfl * self.h / torch.maximum(vlen[s], c), self.h / vlen[s])
            best = min(best, float(dt.min()))
        return math.floor(best * 1.0e12) / 1.0e12

    def positions(self):
        out = np.zeros((len(self.x), 4))
        out[:, : self.dim] = self.x.cpu().numpy()
        return out

    def records(self):
        d, n = self.dim, len(self.x)
        pos, vel = np.zeros((n, 3)), np.zeros((n, 3))
        pos[:, :d], vel[:, :d] = self.x.cpu().numpy(), self.v.cpu().numpy()
        F, C = np.zeros((n, 3, 3)), np.zeros((n, 3, 3))
        F[:, :d, :d] = self.F.cpu().numpy().transpose(0, 2, 1)
        C[:, :d, :d] = self.C.cpu().numpy().transpose(0, 2, 1)
        return {"position": pos, "velocity": vel, "def_grad": F.reshape(n, 9), "affine": C.reshape(n, 9),
                "plastic": self.model[:, :3].cpu().numpy(), "enabled": None}


def _rotation(q, d):
    if d == 2:
        return np.array([[q[0], -q[1]], [q[1], q[0]]])
    x, y, z, w = q
    return np.array([
        [1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
        [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
        [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)],
    ])


def _spin(q, rv):
    """The quaternion (i, j, k, w) turned by the rotation vector rv."""
    ang = np.linalg.norm(rv)
    v, w = (rv * (math.sin(ang / 2) / ang), math.cos(ang / 2)) if ang > 0 else (np.zeros(3), 1.0)
    out = np.empty(4)
    out[:3] = w * q[:3] + q[3] * v + np.cross(v, q[:3])
    out[3] = w * q[3] - v @ q[:3]
    return out * 0.5 * (3.0 - out @ out)


def _exact_of(sc):
    return _Exact(sc.particles, sc.bodies, sc.cell_width, sc.params, sc.dim)


def exact(case, seed):
    kind = case["kind"]
    if kind == "served":  # hundreds of substeps of many scenes: over 20 seconds
        return None
    if kind == "batch":
        if case["scenes"] * case["substeps"] > 1000:
            return None
        outs = []
        for sc in _scene_list(case, seed, case["scenes"]):
            ex = _exact_of(sc)
            for _ in range(case["substeps"]):
                ex.step()
            outs.append(ex.positions())
        return {"positions": np.concatenate(outs)}
    if kind == "emitter":
        pool, layer = _emitter(case, seed)
        ex = _exact_of(pool)
        ex.append(layer)
        for _ in range(case["substeps"]):
            ex.step()
        return {"positions": ex.positions()[len(layer) :]}
    sc = _scene(case, seed)
    ex = _exact_of(sc)
    if kind == "adaptive":
        bound = ex.timestep_bound()
        n = adaptive_substeps(case["frame_dt"], bound, 1, 40)
        ex.dt = _f32(case["frame_dt"] / n)
        for _ in range(n):
            ex.step()
        return {**ex.records(), "bound": bound}
    for _ in range(case["substeps"]):
        ex.step()
    if kind == "frame" and not case["full"]:
        return {"positions": ex.positions()}
    res = ex.records()
    if kind == "frame":
        tra, lin = np.zeros((len(ex.bodies), 4)), np.zeros((len(ex.bodies), 4))
        for i, b in enumerate(ex.bodies):
            tra[i, : ex.dim], tra[i, 3] = b["tra"], b["scale"]
            lin[i, :3] = b["lin"]
        res["translation"], res["linvel"] = tra, lin
    return res
