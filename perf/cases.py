"""The work that programs have this library do, as measurable cases.

Every case goes through the package's public entry points (cup3d_b200.Context
and cup3d_b200.Batch) on device-resident fields, as a host program that keeps
its fields on the GPU does.  Kinds:

  box_step     one cup_step of a uniform periodic box (Taylor-Green class flow)
  sphere_step  one cup_step of the flow past a sphere on its refined mesh
  swarm_step   one cup_batch_step of independent moving ellipsoids
  solve        one Poisson solve from zero on the sphere mesh
  advect       AdvectionDiffusion alone, on the sphere mesh or on a box
  project      the projection's two stencil passes around a given increment
  inverse      the device inverse that the two-level coarse space is built with
  train        Adam steps of the learned preconditioner's network

Step and operator cases put their initial fields back with device copies on
the context's stream before each pass, so that every pass does the same work.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cup3d_b200 as cup
from cup3d_b200 import _lib
from cup3d_b200.workloads import (SPHERE_BODY, SPHERE_FLAGS, SPHERE_MESH, SPHERE_RE1000_FLAGS,
                                  make_swarm_ctx)

STEP = 200  # past the CFL ramp, with the previous pressure in the right-hand side


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: the 32^3 Taylor-Green vortex, 64 blocks, where
        # launches, barriers and latency are the time
        {"name": "tgv32_step", "kind": "box_step", "bx": 4, "by": 4, "bz": 4, "advection": "upwind5"},
        # the library's benchmark step: sphere at Re=300, 2340 blocks
        {"name": "sphere_step", "kind": "sphere_step", "level_max": 4, "wake": 3.0, "solver": "b200_twolevel"},
        # the larger single case: Re=1000, one level finer, 5000 blocks
        {"name": "sphere_fine_step", "kind": "sphere_step", "level_max": 5, "wake": 3.0, "solver": "b200_twolevel"},
        # many independent cases with moving bodies in one batch (the largest case)
        {"name": "swarm16_step", "kind": "swarm_step", "cases": 16, "first": 0},
        # the Poisson solve by itself, as PoissonSolverBase::solve() is called:
        # the default solver, the two-level one in mixed precision, and the
        # two-level one to a tight tolerance
        {"name": "solve_plain", "kind": "solve", "level_max": 4, "wake": 3.0, "solver": "b200", "tol": 1e-6},
        {"name": "solve_twolevel_mixed", "kind": "solve", "level_max": 4, "wake": 3.0,
         "solver": "b200_twolevel_mixed", "tol": 1e-6},
        {"name": "solve_twolevel_tight", "kind": "solve", "level_max": 4, "wake": 3.0, "solver": "b200_twolevel",
         "tol": 1e-10},
        # the operators that a host program calls one by one
        {"name": "advect_weno5_sphere", "kind": "advect", "mesh": "sphere", "level_max": 4, "wake": 3.0,
         "advection": "weno5"},
        {"name": "advect_upwind5_box", "kind": "advect", "mesh": "box", "bx": 13, "by": 11, "bz": 15,
         "advection": "upwind5", "bc": "mixed"},
        {"name": "project_sphere", "kind": "project", "level_max": 4, "wake": 3.0},
        # the coarse space's inverse, once per mesh adaptation and per batch case
        {"name": "inverse_604", "kind": "inverse", "n": 604},
        # forward, backward and update of the learned preconditioner's network
        {"name": "train_128", "kind": "train", "batch": 128, "steps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box_step", "sphere_step", "swarm_step", "solve", "advect", "advect", "project", "inverse",
                       "train"])
    sphere = {"level_max": rng.choice([3, 4, 4, 5]), "wake": round(rng.uniform(1.0, 3.2), 2)}
    if kind == "box_step":
        return {"kind": kind, "bx": rng.randint(2, 8), "by": rng.randint(2, 8), "bz": rng.randint(2, 9),
                "advection": rng.choice(["upwind5", "weno5"])}
    if kind == "sphere_step":
        return dict(sphere, kind=kind, solver=rng.choice(["b200_twolevel", "b200_twolevel", "b200"]))
    if kind == "swarm_step":
        return {"kind": kind, "cases": _log_int(rng, 2, 14), "first": rng.randint(0, 40)}
    if kind == "solve":
        solver = rng.choice(["b200", "b200_twolevel", "b200_twolevel_mixed"])
        return dict(sphere, kind=kind, level_max=rng.choice([3, 4]), solver=solver,
                    tol=1e-10 if solver == "b200_twolevel" else 1e-6)
    if kind == "advect":
        scheme = rng.choice(["upwind5", "weno5"])
        if rng.random() < 0.5:
            return dict(sphere, kind=kind, mesh="sphere", advection=scheme)
        n = [_log_int(rng, 2, 16) for _ in range(3)]
        return {"kind": kind, "mesh": "box", "bx": n[0], "by": n[1], "bz": n[2], "advection": scheme,
                "bc": rng.choice(["periodic", "mixed"])}
    if kind == "project":
        return dict(sphere, kind=kind)
    if kind == "inverse":
        return {"kind": kind, "n": _log_int(rng, 33, 1400)}
    return {"kind": kind, "batch": _log_int(rng, 24, 384), "steps": rng.randint(5, 20)}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return np.random.Generator(np.random.PCG64([int(seed) & 0x7FFFFFFF, salt]))


def _centres(ctx):
    """Cell centres (nb*512, 3) and spacings (nb*512,) on the GPU, in block order."""
    _, index, h = ctx.blocks()
    idx = torch.tensor(index, device="cuda", dtype=torch.float64)
    hh = torch.tensor(h, device="cuda")
    c = torch.arange(512, device="cuda")
    cell = torch.stack([c % 8, (c // 8) % 8, c // 64], 1).double() + 0.5
    xyz = (idx[:, None, :] * 8 + cell[None]) * hh[:, None, None]
    return xyz.reshape(-1, 3), hh.repeat_interleave(512)


def _modes(xyz, lengths, g, amp, count=5, top=3):
    """Smooth periodic velocity: TGV-like base flow plus seeded divergence-free
    Fourier modes, (3, n)."""
    w = [2 * math.pi / L for L in lengths]
    x, y, z = (xyz[:, d] * w[d] for d in range(3))
    u = torch.stack([torch.sin(x) * torch.cos(y) * torch.cos(z),
                     -(w[0] / w[1]) * torch.cos(x) * torch.sin(y) * torch.cos(z), 0 * z])
    for _ in range(count):
        k = g.integers(-top, top + 1, 3)
        if not k.any():
            k[2] = 1
        kw = np.array([k[d] * w[d] for d in range(3)])
        a = np.cross(kw, g.standard_normal(3))
        a *= amp / max(np.linalg.norm(a), 1e-12)
        ph = float(k[0]) * x + float(k[1]) * y + float(k[2]) * z + float(g.uniform(0, 2 * math.pi))
        u += torch.tensor(a, device=xyz.device)[:, None] * torch.cos(ph)[None]
    return u


def _vortices(xyz, g, centre, spread, radius, amp, count=12):
    """Velocity of seeded Gaussian vortices (curl of a vector potential) near a
    body and its wake, (3, n)."""
    u = torch.zeros(3, xyz.shape[0], dtype=torch.float64, device=xyz.device)
    for _ in range(count):
        c = torch.tensor(np.asarray(centre) + spread * g.uniform(-1, 1, 3), device=xyz.device)
        r = radius * g.uniform(1.0, 3.0)
        a = g.standard_normal(3)
        a *= amp / np.linalg.norm(a)
        d = (xyz - c) / r
        e = torch.exp(-0.5 * (d * d).sum(1))
        u += torch.stack([a[1] * d[:, 2] - a[2] * d[:, 1], a[2] * d[:, 0] - a[0] * d[:, 2],
                          a[0] * d[:, 1] - a[1] * d[:, 0]]) * e[None]
    return u


def _bumps(xyz, h, g, centre, spread, amp, count=8):
    """Sum of seeded Gaussian sources a few cells to many cells wide."""
    out = torch.zeros(xyz.shape[0], dtype=torch.float64, device=xyz.device)
    for _ in range(count):
        c = torch.tensor(np.asarray(centre) + spread * g.uniform(-1, 1, 3), device=xyz.device)
        d2 = ((xyz - c) ** 2).sum(1)
        sigma = float(g.uniform(2.0, 8.0)) * float(h[int(torch.argmin(d2))])
        out += amp * float(g.standard_normal()) * torch.exp(-d2 / (2 * sigma * sigma))
    return out


class _Array:
    """Device memory of a context's field, for torch (zero copy)."""

    def __init__(self, ctx, ptr, n):
        self.ctx = ctx  # the memory is the context's
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


class _State:
    """A context, its stream and the fields that every pass starts from."""

    def __init__(self, case, ctx):
        self.case, self.ctx = case, ctx
        self.stream = torch.cuda.ExternalStream(int(_lib.lib().cup_stream(ctx._p)))
        self.views, self.saved, self.more = {}, {}, {}

    def field(self, name):
        ptr = self.ctx.field_ptr(name)  # fields are double-buffered: asked for on each pass
        if ptr not in self.views:
            self.views[ptr] = torch.as_tensor(_Array(self.ctx, ptr, _lib.FIELD_NCOMP[name] * self.ctx.nb * 512),
                                              device="cuda")
        return self.views[ptr]

    def keep(self, name, value):
        self.saved[name] = value.reshape(-1).contiguous()

    def restore(self, *names):
        with torch.cuda.stream(self.stream):
            for n in names:
                self.field(n).copy_(self.saved[n])


def _box(case, extra=""):
    bc = "periodic periodic periodic" if case.get("bc", "periodic") == "periodic" else "periodic wall freespace"
    bcx, bcy, bcz = bc.split()
    top = max(case["bx"], case["by"], case["bz"])
    cfg = cup.config(f"-bpdx {case['bx']} -bpdy {case['by']} -bpdz {case['bz']} -levelMax 1 "
                     f"-extent {2 * math.pi * top / 4!r} -nu 0.01 -CFL 0.3 -BC_x {bcx} -BC_y {bcy} -BC_z {bcz} "
                     f"-advection {case['advection']} -poissonTol 0 -poissonTolRel 1e-8 {extra}",
                     device=0)
    ctx = cup.Context(cfg)
    ctx.set_mesh_uniform()
    return ctx


def _box_lengths(case):
    return [case[k] * math.pi / 2 for k in ("bx", "by", "bz")]


def _sphere(case, extra=""):
    flags = SPHERE_FLAGS if case["level_max"] < 5 else SPHERE_RE1000_FLAGS
    flags = flags.replace("-levelMax 4", f"-levelMax {case['level_max']}")
    ctx = cup.Context(cup.config(f"{flags} {extra}", device=0))
    ctx.set_mesh_sphere_wake(**dict(SPHERE_MESH, wake_radius=case["wake"]))
    return ctx


def _sphere_flow(xyz, seed):
    c = np.array(SPHERE_BODY["center"]) - np.array([0.2, 0.0, 0.0])
    return _vortices(xyz, _gen(seed, 1), c, np.array([0.3, 0.1, 0.1]), SPHERE_BODY["radius"], 0.05)


def _pressure(xyz, h, seed, amp=1e-3):
    g = _gen(seed, 2)
    return _bumps(xyz, h, g, SPHERE_BODY["center"], np.array([0.4, 0.2, 0.2]), amp)


def _zero_mean(v, h):
    w = h ** 3
    return v - (v * w).sum() / w.sum()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "box_step":
        s = _State(case, _box(case))
        xyz, _ = _centres(s.ctx)
        s.keep("vel", _modes(xyz, _box_lengths(case), _gen(seed, 1), 0.3))
        s.keep("pres", 0.1 * _modes(xyz, _box_lengths(case), _gen(seed, 2), 0.3)[0])
        for _ in range(2):  # the program has stepped before
            run(s)
        return s
    if kind == "sphere_step":
        s = _State(case, _sphere(case, f"-poissonSolver {case['solver']}"))
        s.ctx.obstacle_sphere(**SPHERE_BODY)
        xyz, h = _centres(s.ctx)
        s.keep("vel", _sphere_flow(xyz, seed))
        s.keep("pres", _pressure(xyz, h, seed))
        for _ in range(2):
            run(s)
        return s
    if kind == "swarm_step":
        cases = []
        for i in range(case["first"], case["first"] + case["cases"]):
            c = make_swarm_ctx(i, 0, "-poissonSolver b200_twolevel -StaticObstacles 0")
            xyz, h = _centres(c)
            t = _State(case, c)
            t.keep("vel", _modes(xyz, [1.0, 1.0, 1.0], _gen(seed, 100 + i), 0.05) * 0.1)
            t.keep("pres", _bumps(xyz, h, _gen(seed, 500 + i), (0.5, 0.5, 0.5), np.full(3, 0.2), 1e-3))
            t.restore("vel", "pres")
            t.stream.synchronize()
            cases.append(c)
        s = _State(case, cup.Batch(cases))
        for n in ("vel", "pres"):
            s.keep(n, s.field(n).clone())
        torch.cuda.synchronize()
        for c in cases:
            c.close()
        return s
    if kind == "solve":
        s = _State(case, _sphere(case))
        s.ctx.set_poisson(case["solver"], 0.0, case["tol"], 1000)
        xyz, h = _centres(s.ctx)
        if case["tol"] < 1e-8:
            x = _solution(xyz, h, seed)
            b = torch.empty_like(x)
            torch.cuda.synchronize()
            s.ctx.poisson_apply(x, b)
        else:
            g = _gen(seed, 3)
            noise = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
            b = torch.randn(h.shape[0], dtype=torch.float64, device="cuda", generator=noise)
            spread = np.full(3, SPHERE_BODY["radius"] + 0.5)
            b = _zero_mean(b + _bumps(xyz, h, g, SPHERE_BODY["center"], spread, 10.0), h)
        s.more = {"b": b.contiguous(), "x": torch.zeros_like(b)}
        torch.cuda.synchronize()
        if "twolevel" in case["solver"]:  # the mesh's coarse space, kept as long as the mesh
            s.ctx.coarse_apply(s.more["b"], s.more["x"])
        return s
    if kind == "advect":
        if case["mesh"] == "box":
            s = _State(case, _box(case))
            xyz, h = _centres(s.ctx)
            s.keep("vel", _modes(xyz, _box_lengths(case), _gen(seed, 1), 0.3))
            s.more["dt"] = 0.02
        else:
            s = _State(case, _sphere(case, f"-advection {case['advection']}"))
            xyz, h = _centres(s.ctx)
            s.keep("vel", _sphere_flow(xyz, seed))
            s.more["dt"] = 0.5 * float(h.min())
        return s
    if kind == "project":
        s = _State(case, _sphere(case))
        s.ctx.obstacle_sphere(**SPHERE_BODY)
        xyz, h = _centres(s.ctx)
        s.keep("vel", _sphere_flow(xyz, seed))
        s.keep("pres", _pressure(xyz, h, seed))
        s.more = {"phi": _pressure(xyz, h, int(seed) + 77, 1e-4), "dt": 0.5 * float(h.min())}
        return s
    if kind == "inverse":
        n = case["n"]
        ctx = cup.Context(cup.config("-bpdx 1 -bpdy 1 -bpdz 1", device=0))
        ctx.set_mesh_uniform()
        s = _State(case, ctx)
        s.more = {"a0": _coarse_like(n, seed)}
        s.more["a"] = s.more["a0"].clone()
        return s
    # train: samples of the solver's residuals on a box of 256 blocks
    s = _State(case, _box({"bx": 8, "by": 8, "bz": 4, "advection": "upwind5", "bc": "mixed"}))
    s.ctx.cnn_init(int(seed) & 0xFFFF)
    s.more["params"] = s.ctx.cnn_get_params()
    xyz, h = _centres(s.ctx)
    s.ctx.cnn_dataset_reserve(4 * s.ctx.nb)
    noise = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    mid = np.array(_box_lengths({"bx": 8, "by": 8, "bz": 4})) / 2
    for k in range(4):
        r = _bumps(xyz, h, _gen(seed, 20 + k), mid, mid, 1.0, 24)
        r += 0.05 * torch.randn(r.shape[0], dtype=torch.float64, device="cuda", generator=noise)
        torch.cuda.synchronize()
        s.ctx.cnn_dataset_add(r.contiguous())
    return s


def _solution(xyz, h, seed):
    """A solution with the smooth and the rough parts a pressure has, zero mean."""
    noise = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    x = _bumps(xyz, h, _gen(seed, 3), SPHERE_BODY["center"], np.array([0.6, 0.3, 0.3]), 1.0)
    x += 0.01 * torch.randn(x.shape[0], dtype=torch.float64, device="cuda", generator=noise)
    return _zero_mean(x, h).contiguous()


def _coarse_like(n, seed):
    """A matrix with the make of a coarse operator: the weighted graph Laplacian
    of a 3-D arrangement of n blocks, and one row of volume weights."""
    g = _gen(seed, 4)
    a = np.zeros((n, n))
    m = max(2, int(round(n ** (1 / 3))))
    for s in (1, m, m * m):
        i = np.arange(n - s)
        if len(i):
            w = np.exp2(g.integers(0, 3, len(i))) * g.uniform(0.5, 1.5, len(i))
            a[i, i + s] += w
            a[i + s, i] += w
    a[np.arange(n), np.arange(n)] = -a.sum(1) - 1e-3 * a.sum(1).mean()
    a[n // 3] = g.uniform(0.2, 1.0, n)
    return torch.tensor(a, device="cuda")


# -------------------------------------------------------------------- runs
def run(s):
    kind, ctx = s.case["kind"], s.ctx
    if kind in ("box_step", "sphere_step"):
        s.restore("vel", "pres")
        dt, _, _ = ctx.step(STEP)
        return {"vel": s.field("vel"), "pres": s.field("pres"), "dt": dt}
    if kind == "swarm_step":
        s.restore("vel", "pres")
        _, dt, force, _ = ctx.step(STEP)
        return {"vel": s.field("vel"), "pres": s.field("pres"), "dt": dt, "force": force}
    if kind == "solve":
        with torch.cuda.stream(s.stream):
            s.more["x"].zero_()
        ctx.poisson_solve_dev(s.more["b"], s.more["x"])
        return s.more["x"]
    if kind == "advect":
        s.restore("vel")
        ctx.advect_diffuse(s.more["dt"])
        return s.field("vel")
    if kind == "project":
        s.restore("vel", "pres")
        ctx.pressure_rhs(s.more["dt"], STEP)
        with torch.cuda.stream(s.stream):  # the increment, in the solve's place
            s.field("pres").copy_(s.more["phi"])
        ctx.pressure_finish(s.more["dt"], STEP)
        return {"rhs": s.field("lhs"), "vel": s.field("vel"), "pres": s.field("pres")}
    if kind == "inverse":
        with torch.cuda.stream(s.stream):
            s.more["a"].copy_(s.more["a0"])
        ctx.dense_inverse(s.more["a"], s.case["n"] // 3)
        return s.more["a"]
    ctx.cnn_set_params(s.more["params"])  # the same start on each pass, moments zeroed
    losses = ctx.cnn_train(s.case["steps"], s.case["batch"], 1e-3, 7)
    return {"losses": losses, "params": ctx.cnn_get_params()}


# ------------------------------------------------------------------- work
_BLOCKS = {}


def _cells(case):
    if "bx" in case:
        return 512 * case["bx"] * case["by"] * case["bz"]
    key = tuple(sorted((k, v) for k, v in case.items() if k in ("level_max", "wake", "cases", "first")))
    if key not in _BLOCKS:
        if "cases" in case:
            n = 0
            for i in range(case["first"], case["first"] + case["cases"]):
                with make_swarm_ctx(i, -1) as c:
                    n += c.nb
        else:
            flags = SPHERE_FLAGS.replace("-levelMax 4", f"-levelMax {case['level_max']}")
            with cup.Context(cup.config(flags, device=-1)) as c:
                c.set_mesh_sphere_wake(**dict(SPHERE_MESH, wake_radius=case["wake"]))
                n = c.nb
        _BLOCKS[key] = n
    return 512 * _BLOCKS[key]


def work(case):
    """Each field read once and written once; the arithmetic of the advection
    (9 face reconstructions or derivatives a cell and stage) and of one
    application of the operator and the block inverse (a step's or a solve's
    iterations are the method's own affair)."""
    kind = case["kind"]
    if kind == "inverse":
        return {"bytes": 16 * case["n"] ** 2, "flops": 2 * case["n"] ** 3}
    if kind == "train":
        # per sample: the input and target; forward, input gradient and weight
        # gradient of two 16 x 16 and two 1 x 16 channel 3^3 convolutions
        per = 3 * 2 * 27 * (2 * 256 * 512 + 2 * 16 * 512)
        return {"bytes": case["steps"] * case["batch"] * (1000 + 512) * 4, "flops": case["steps"] * case["batch"] * per}
    n = _cells(case)
    adv = 3 * 9 * (70 if case.get("advection", "weno5") == "weno5" else 14) + 3 * 3 * 10
    if kind == "advect":
        return {"bytes": 48 * n, "flops": n * adv}
    if kind == "project":
        return {"bytes": (24 + 8 + 8 + 8 + 24 + 8) * n, "flops": 50 * n}
    if kind == "solve":
        return {"bytes": 16 * n, "flops": 120 * n}
    return {"bytes": 64 * n, "flops": n * (adv + 50 + 120)}


def tolerance(case):
    """About four times what the path shows against itself: with its inputs
    moved by one rounding, with its sums in another order, and where a solve
    ends the pass, with the stopping test passed one iteration sooner or later."""
    kind = case["kind"]
    if kind == "box_step":  # solved to 1e-8: pressure 6e-8, largest 3e-7
        return {"rel": 3e-7, "max": 2e-6}
    if kind in ("sphere_step", "swarm_step"):  # solved to 1e-4: pressure 9e-4, largest 3e-3
        return {"rel": 4e-3, "max": 1.5e-2}
    if kind == "solve":  # 7e-6 and 1.4e-5 at 1e-6; 5e-9 and 1.2e-8 at 1e-10
        return {"rel": 2e-8, "max": 5e-8} if case["tol"] < 1e-8 else {"rel": 3e-5, "max": 8e-5}
    if kind == "advect":  # 64-bit stencils: 4e-16 and 1e-15 for moved inputs; WENO5's weights amplify more
        return {"rel": 1e-13, "max": 1e-12}
    if kind == "project":  # the right-hand side is a difference of large terms: 5e-13 and 1.7e-11
        return {"rel": 2e-12, "max": 7e-11}
    if kind == "inverse":  # 2e-15 and 2e-14 at n = 604, growing with the condition
        return {"rel": 1e-12, "max": 1e-11}
    # 16-bit activations under 32-bit sums: 3e-5 and 4e-4 for moved weights; a
    # sum in another order also moves the activations' roundings
    return {"rel": 5e-4, "max": 5e-3}


# ------------------------------------------------------ results in 64 bits
def _lattice(case):
    """For each cell of the box in device order, its index in a [z][y][x]
    array (the device's block order is asked of the mesh; host only)."""
    cfg = cup.config(f"-bpdx {case['bx']} -bpdy {case['by']} -bpdz {case['bz']} -levelMax 1", device=-1)
    with cup.Context(cfg) as ctx:
        ctx.set_mesh_uniform()
        index = torch.tensor(ctx.blocks()[1], device="cuda", dtype=torch.int64)
    c = torch.arange(512, device="cuda")
    cell = torch.stack([c % 8, (c // 8) % 8, c // 64], 1)
    p = (index[:, None, :] * 8 + cell[None]).reshape(-1, 3)
    return (p[:, 2] * 8 * case["by"] + p[:, 1]) * 8 * case["bx"] + p[:, 0], p


def _pad(u, c, axis, bc, layers=3):
    """u (grid [z][y][x], component c) with ghost layers along one axis."""
    d = 2 - axis  # coordinate of the array axis
    if bc[d] == "periodic":
        return torch.cat([u.narrow(axis, u.shape[axis] - layers, layers), u, u.narrow(axis, 0, layers)], axis)
    sign = -1.0 if bc[d] == "wall" or c == d else 1.0
    lo, hi = u.narrow(axis, 0, 1), u.narrow(axis, u.shape[axis] - 1, 1)
    rep = [layers if a == axis else 1 for a in range(3)]
    return torch.cat([sign * lo.repeat(rep), u, sign * hi.repeat(rep)], axis)


def _weno(a, b, c, d, e):
    b1 = 13 / 12 * (a + c - 2 * b) ** 2 + 0.25 * (a + 3 * c - 4 * b) ** 2
    b2 = 13 / 12 * (b + d - 2 * c) ** 2 + 0.25 * (b - d) ** 2
    b3 = 13 / 12 * (c + e - 2 * d) ** 2 + 0.25 * (3 * c + e - 4 * d) ** 2
    w = [0.1 / (b1 + 1e-6) ** 2, 0.6 / (b2 + 1e-6) ** 2, 0.3 / (b3 + 1e-6) ** 2]
    f = [11 / 6 * c + a / 3 - 7 / 6 * b, 5 / 6 * c - b / 6 + d / 3, c / 3 + 5 / 6 * d - e / 6]
    return (w[0] * f[0] + w[1] * f[1] + w[2] * f[2]) / (w[0] + w[1] + w[2])


def _advected(u, scheme, bc, h, dt, nu):
    """AdvectionDiffusion of u (3 grids) with the low-storage RK3."""
    u, tmp = list(u), [0.0, 0.0, 0.0]
    for alpha, beta in ((1 / 3, -5 / 9), (15 / 16, -153 / 128), (8 / 15, 0.0)):
        rhs = []
        for c in range(3):
            r = 0.0
            for axis in range(3):
                v, n = _pad(u[c], c, axis, bc), u[c].shape[axis]
                m3, m2, m1, u0, p1, p2, p3 = (v.narrow(axis, 3 + k, n) for k in range(-3, 4))
                U = u[2 - axis]
                if scheme == "weno5":
                    plus = _weno(m2, m1, u0, p1, p2) - _weno(m3, m2, m1, u0, p1)
                    minus = _weno(p3, p2, p1, u0, m1) - _weno(p2, p1, u0, m1, m2)
                else:
                    plus = (-2 * m3 + 15 * m2 - 60 * m1 + 20 * u0 + 30 * p1 - 3 * p2) / 60
                    minus = (2 * p3 - 15 * p2 + 60 * p1 - 20 * u0 - 30 * m1 + 3 * m2) / 60
                r = r - dt / h * U * torch.where(U > 0, plus, minus) + nu * dt / (h * h) * (p1 + m1 - 2 * u0)
            rhs.append(r)
        tmp = [tmp[c] + rhs[c] for c in range(3)]
        u = [u[c] + alpha * tmp[c] for c in range(3)]
        tmp = [beta * t for t in tmp]
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "inverse":
        return torch.linalg.inv(_coarse_like(case["n"], seed))
    if kind == "solve" and case["tol"] < 1e-8:
        # the right-hand side was made from this solution
        flags = SPHERE_FLAGS.replace("-levelMax 4", f"-levelMax {case['level_max']}")
        with cup.Context(cup.config(flags, device=-1)) as c:  # the cells' places, host only
            c.set_mesh_sphere_wake(**dict(SPHERE_MESH, wake_radius=case["wake"]))
            xyz, h = _centres(c)
        return _solution(xyz, h, seed)
    if kind == "box_step" or (kind == "advect" and case["mesh"] == "box"):
        at, p = _lattice(case)
        top = max(case["bx"], case["by"], case["bz"])
        h = 2 * math.pi * top / 4 / (8 * top)
        xyz = (p.double() + 0.5) * h
        shape = (8 * case["bz"], 8 * case["by"], 8 * case["bx"])
        back = torch.empty_like(at)
        back[at] = torch.arange(at.numel(), device="cuda")
        grid = lambda v: v[back].reshape(shape)  # noqa: E731
        u = [grid(v) for v in _modes(xyz, _box_lengths(case), _gen(seed, 1), 0.3)]
        bc = ("periodic",) * 3 if case.get("bc", "periodic") == "periodic" else ("periodic", "wall", "freespace")
        if kind == "advect":
            u = _advected(u, case["advection"], bc, h, 0.02, 0.01)
            return torch.stack([v.reshape(-1)[at] for v in u]).reshape(-1)
        umax = max(float(v.abs().max()) for v in u)
        dt = min(h * h / 6 / (0.01 + h / 6 * umax), 0.3 * h / (umax + 1e-8))
        pold = grid(0.1 * _modes(xyz, _box_lengths(case), _gen(seed, 2), 0.3)[0])
        u = _advected(u, case["advection"], bc, h, dt, 0.01)
        roll = lambda v, axis: (torch.roll(v, -1, axis), torch.roll(v, 1, axis))  # noqa: E731
        div = sum(roll(u[c], 2 - c)[0] - roll(u[c], 2 - c)[1] for c in range(3)) * (0.5 * h * h / dt)
        lap = h * (sum(sum(roll(pold, a)) for a in range(3)) - 6 * pold)
        k = [2 - 2 * torch.cos(2 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n) for n in shape]
        lam = -h * (k[0][:, None, None] + k[1][None, :, None] + k[2][None, None, :])
        lam[0, 0, 0] = 1.0
        f = torch.fft.fftn(div - lap) / lam
        f[0, 0, 0] = 0.0
        pres = torch.fft.ifftn(f).real + pold
        u = [u[c] - 0.5 * dt / h * (roll(pres, 2 - c)[0] - roll(pres, 2 - c)[1]) for c in range(3)]
        return {"vel": torch.stack([v.reshape(-1)[at] for v in u]).reshape(-1), "pres": pres.reshape(-1)[at],
                "dt": dt}
    # A refined mesh's stencils use the library's own interpolation across
    # levels, a solve to 1e-6 ends where its stopping test lets it, and the
    # training draws its samples inside the library: no plain form of these.
    return None
