"""The work that users have this library do, as cases that can be timed.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (a context some frames into its flow, device arrays, a network),
`run` makes one pass through the public entry points and returns its outputs,
`work` says what that pass cannot do without, and `exact` evaluates the pass in
64 bits with torch alone.

Kinds of case:
  passes  the ComputeStep sequence driven pass by pass, as the headless
          harnesses and a host that records its own command list do
  app     one application frame through FrameDriver: parameters in, a
          neighbour search, the substeps of 1/60 s, stats out, positions for
          the renderer
  frames  whole device-resident frames (fe_step) of a dam break, with the
          positions and velocities copied out asynchronously
  batch   the same over many scenes in one context
  sort    the standalone sort of device key/value pairs
  water   density splat + water pass, image copied out
  train   training steps of the warm-start network
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fluid-engine_b200"))

from fluid_step import _abi, camera, frame, scene  # noqa: E402
from fluid_step.learned import Model  # noqa: E402
from fluid_step.pipelines import (BatchSimulation, CommandBufferBuilder,  # noqa: E402
                                  ComputePipelines, GpuPhysicsData, Simulation)

SPACING = 0.05      # of the dam breaks; h = 0.1
APP_SPACING = 0.04  # of the application's and the harnesses' scenes; h = 0.08
PAIRS = 31          # neighbours per particle in the bulk of these flows

# Mean and deviation of the 12 features and 2 targets over captures of the 16k
# and 262k dam breaks (what training finds); the cases' networks are drawn
# around them, so that their starts are of the size a trained one gives.
X_MEAN = [-0.0805, 115.6, -0.759, 0.8065, 5.593, 6.122, 0.0346, -0.4415, 0.4648, -0.3537,
          0.3475, -0.2879]
X_STD = [0.1307, 31.56, 7.638, 0.1946, 16.74, 15.08, 0.0431, 0.4388, 0.2938, 0.3334, 0.2817,
         0.2943]
Y_MEAN = [5.622, 0.6562]
Y_STD = [16.82, 11.32]


def listed():
    return [
        # The convergence harness: 4800 particles (20 x 20 x 12), bitonic
        # sort, ten substeps recorded pass by pass in one submit.
        {"name": "harness_4800", "kind": "passes", "nx": 20, "ny": 20, "nz": 12, "sort": "bitonic",
         "iters": 4, "substeps": 10},
        # The application's frame: its 25k-particle scene, moving wall,
        # 4 substeps of 5 ms with 4 + 4 iterations.
        {"name": "app_25k", "kind": "app", "nx": 25, "ny": 50, "nz": 20},
        # Single frames of a small scene, 4 + 4 iterations: launches count.
        {"name": "frame_16k", "kind": "frames", "nx": 16, "ny": 32, "nz": 32, "mode": "reference",
         "solver": "fixed", "cfl": 0.0, "learned": False, "warm": 2},
        # Interactive size under the adaptive step: the pressure solve
        # iterates to 0.1 %, some 15 iterations a frame.
        {"name": "frame_262k_cfl", "kind": "frames", "nx": 64, "ny": 64, "nz": 64, "mode": "fixed",
         "solver": "tolerance", "cfl": 0.3, "learned": False, "warm": 150},
        # The same with the learned warm start: features, network, carried state.
        {"name": "frame_262k_learned", "kind": "frames", "nx": 64, "ny": 64, "nz": 64,
         "mode": "fixed", "solver": "tolerance", "cfl": 0.3, "learned": True, "warm": 60},
        # The headline: 1M particles, dt 1 ms, tolerance 0.1 %.
        {"name": "frame_1m", "kind": "frames", "nx": 128, "ny": 64, "nz": 128, "mode": "fixed",
         "solver": "tolerance", "cfl": 0.0, "learned": False, "warm": 6},
        # The largest scene.
        {"name": "frame_4m", "kind": "frames", "nx": 256, "ny": 64, "nz": 256, "mode": "fixed",
         "solver": "tolerance", "cfl": 0.0, "learned": False, "warm": 6},
        # Many small scenes in one context.
        {"name": "batch_256", "kind": "batch", "scenes": 256, "lo": 1024, "hi": 8192, "warm": 2},
        # The standalone sort: a small and a large array of random keys.
        {"name": "sort_32k", "kind": "sort", "n": 32768, "key_bits": 32, "algorithm": "radix"},
        {"name": "sort_4m", "kind": "sort", "n": 4194304, "key_bits": 32, "algorithm": "radix"},
        # A frame's rendering: splat into 128^3 and shade 1280 x 720.
        {"name": "water_262k", "kind": "water", "nx": 64, "ny": 64, "nz": 64, "rx": 128, "ry": 128,
         "rz": 128, "width": 1280, "height": 720, "warm": 40},
        # An epoch's stretch of training: 24 steps of 4096 samples.
        {"name": "train_4096", "kind": "train", "batch": 4096, "steps": 24},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def block(lo, hi):
        """Lattice counts of about a log-uniform number of particles."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
        nx = max(4, int(round((n * a * b) ** (1 / 3))))
        ny = max(4, int(round(nx / a)))
        return {"nx": nx, "ny": ny, "nz": max(4, int(round(n / (nx * ny))))}

    kind = rng.choice(["passes", "app", "frames", "frames", "frames", "batch", "sort", "water",
                       "train"])
    if kind == "passes":
        return {"kind": kind, **block(1500, 60000), "sort": rng.choice(["bitonic", "radix"]),
                "iters": rng.randint(3, 8), "substeps": rng.randint(4, 12)}
    if kind == "app":
        return {"kind": kind, **block(6000, 120000)}
    if kind == "frames":
        tol = rng.random() < 0.6
        return {"kind": kind, **block(8000, 2000000), "mode": "fixed" if tol else "reference",
                "solver": "tolerance" if tol else "fixed", "cfl": 0.0,
                "learned": tol and rng.random() < 0.25, "warm": rng.randint(1, 8)}
    if kind == "batch":
        lo = log_int(600, 6000)
        return {"kind": kind, "scenes": log_int(8, 200), "lo": lo, "hi": lo * rng.randint(2, 6),
                "warm": 2}
    if kind == "sort":
        if rng.random() < 0.25:
            return {"kind": kind, "n": 1 << rng.randint(10, 20), "key_bits": 32,
                    "algorithm": "bitonic"}
        return {"kind": kind, "n": log_int(1000, 4000000), "key_bits": rng.choice([32, 32, 20, 13]),
                "algorithm": "radix"}
    if kind == "water":
        return {"kind": kind, **block(16000, 500000), "rx": rng.randint(48, 160),
                "ry": rng.randint(48, 160), "rz": rng.randint(48, 160),
                "width": rng.randint(320, 1600), "height": rng.randint(240, 900),
                "warm": rng.randint(2, 20)}
    return {"kind": "train", "batch": log_int(500, 12000), "steps": rng.randint(4, 32)}


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
def _dam(case, seed):
    """A lattice in a box whose free space grows as the workloads' does."""
    c = (case["nx"], case["ny"], case["nz"])
    n = c[0] * c[1] * c[2]
    side = [2.0 * c[0] * SPACING, 1.25 * c[1] * SPACING, 1.25 * c[2] * SPACING]
    if n == 64 ** 3:
        side = [4.0, 4.0, 4.0]
    if n >= 1 << 20 and c[1] == 64:          # the 1M and 4M dam breaks' boxes
        side = [c[0] / 16.0, 4.0, c[2] / 16.0]
    box = ((0.0, 0.0, 0.0), tuple(float(np.float32(s)) for s in side))
    tol = case.get("solver", "fixed") == "tolerance"
    p = scene.dam_break_params(
        box[0], box[1], use_cfl=case.get("cfl", 0.0) > 0,
        solver=_abi.FE_SOLVER_TOLERANCE if tol else _abi.FE_SOLVER_FIXED_ITERS,
        mode=_abi.FE_MODE_FIXED if case.get("mode") == "fixed" else _abi.FE_MODE_REFERENCE)
    if case.get("cfl", 0.0) > 0:
        p.cfl_lambda = case["cfl"]
    if case.get("learned"):
        p.warm_start = _abi.FE_WARM_LEARNED
    pos, _ = scene.lattice(box[0], c, 0.025, 1000.0, SPACING, 0.01, seed)
    return p, pos


def _app(case, seed):
    """The application's block (Scene::new) in other sizes: the same spacing
    and the box in the same proportions around it."""
    c = (case["nx"], case["ny"], case["nz"])
    f = [c[0] / 25.0, c[1] / 50.0, c[2] / 20.0]
    p = _abi.default_params()
    p.box_min[:] = [float(np.float32(v)) for v in (-1.5 * f[0], 0.0, -1.0 * f[2])]
    p.box_max[:] = [float(np.float32(v)) for v in (0.8 * f[0], 4.0 * f[1], 1.0 * f[2])]
    origin = (-1.0 * f[0], 1.0 * f[1], -0.8 * f[2])
    pos, mass = scene.lattice(origin, c, 0.02, 1000.0, np.float32(APP_SPACING), 0.01, seed)
    p.particle_mass = float(mass)
    return p, pos


def _network(seed):
    rng = np.random.default_rng([seed, 77])
    w1 = np.zeros((64, 16))
    w1[:, :12] = rng.normal(size=(64, 12)) * 0.3
    parts = [w1, rng.normal(size=(64, 64)) * 0.12, rng.normal(size=(2, 64)) * 0.05,
             np.zeros(64), np.zeros(64), np.zeros(2)]
    return np.concatenate([a.reshape(-1) for a in parts]).astype(np.float32)


def _model(seed):
    m = Model(seed=1)
    m.set_normalization(X_MEAN, X_STD, Y_MEAN, Y_STD)
    m.set_parameters(_network(seed))
    return m


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


# ---------------------------------------------------------------------------
# What a program has in hand
# ---------------------------------------------------------------------------
class _Frames:
    """A running simulation whose positions and velocities are copied out
    each frame into page-locked memory, two buffers in turn."""

    def __init__(self, sim, warm, model=None):
        self.sim, self.model = sim, model
        if model is not None:
            lib = sim.data._lib
            _abi.check(lib, lib.fe_set_model(sim.data.handle, model.handle), "fe_set_model")
        n = sim.data.count
        self.out = [(_pinned((n, 4)), _pinned((n, 4))) for _ in range(2)]
        self.turn, self.ticket = 0, None
        for _ in range(warm):
            sim.step(1, want_stats=False)

    def copy_out(self):
        pos, vel = self.out[self.turn]
        self.turn ^= 1
        d = self.sim.data if hasattr(self.sim, "data") else self.sim
        d.download_async(_abi.FE_FIELD_POSITION_A, pos.numpy())
        t = d.download_async(_abi.FE_FIELD_VELOCITY_B, vel.numpy())
        # the frame before this one has arrived by now: its buffers go on
        if self.ticket is not None:
            d.download_wait(self.ticket)
        self.ticket = t
        return pos, vel


def prepare(case, seed):
    kind = case["kind"]
    if kind == "passes":
        p, pos = _app(case, seed)
        p.sort_algorithm = _abi.FE_SORT_BITONIC if case["sort"] == "bitonic" else _abi.FE_SORT_RADIX
        p.density_solver_iterations = p.divergence_solver_iterations = case["iters"]
        data = GpuPhysicsData(pos, p)
        steps = ComputePipelines()
        steps.prepare_all(data, p)
        return {"kind": kind, "data": data, "steps": steps, "first": True,
                "builder": CommandBufferBuilder(data), "iters": case["iters"],
                "substeps": case["substeps"]}
    if kind == "app":
        p, pos = _app(case, seed)
        sim = Simulation(pos, p)
        box = frame.CollisionBox(list(p.box_min), list(p.box_max), 0.3, 0.5)
        f = _Frames(sim, 0)
        f.driver = frame.FrameDriver(sim.data, p, box)
        f.driver.step()
        return {"kind": kind, "frames": f}
    if kind == "frames":
        p, pos = _dam(case, seed)
        f = _Frames(Simulation(pos, p), case["warm"] if not case["learned"] else 0,
                    _model(seed) if case["learned"] else None)
        if case["learned"]:
            for _ in range(case["warm"]):
                f.sim.step(1, want_stats=False)
        return {"kind": kind, "frames": f}
    if kind == "batch":
        w = _batch(case, seed)
        return {"kind": kind, "frames": _Frames(BatchSimulation(w.positions(), w.params()),
                                                case["warm"])}
    if kind == "sort":
        g = torch.Generator().manual_seed(seed)
        n, bits = case["n"], case["key_bits"]
        k = torch.randint(0, 1 << bits, (n,), generator=g, dtype=torch.int64)
        k = torch.where(k >= 1 << 31, k - (1 << 32), k).to(torch.int32).cuda()
        v = torch.arange(n, dtype=torch.int32, device="cuda")
        return {"kind": kind, "keys": k, "vals": v, "k": torch.empty_like(k),
                "v": torch.empty_like(v), "bits": bits, "lib": _abi.load_library(),
                "algorithm": _abi.FE_SORT_RADIX if case["algorithm"] == "radix"
                else _abi.FE_SORT_BITONIC}
    if kind == "water":
        p, pos = _dam(case, seed)
        p.grid_res[:] = [case["rx"], case["ry"], case["rz"]]
        sim = Simulation(pos, p)
        for _ in range(case["warm"]):
            sim.step(1, want_stats=False)
        sim.data.set_skybox(camera.gradient_sky(1024, 512))
        lo, hi = np.asarray(p.box_min), np.asarray(p.box_max)
        mid, size = (lo + hi) / 2, float(np.max(hi - lo))
        cam = camera.make_camera(mid + np.array([0.1, 0.45, -1.25]) * size, mid, case["width"],
                                 case["height"])
        out = [_pinned((case["height"], case["width"], 4)) for _ in range(2)]
        return {"kind": kind, "sim": sim, "cam": cam, "out": out, "turn": 0, "ticket": None}
    x, y = _samples(case, seed)
    return {"kind": "train", "model": _model(seed), "x": x.float().cuda(), "y": y.float().cuda(),
            "batch": case["batch"], "steps": case["steps"]}


def _batch(case, seed):
    w = scene.batch_workload(n_scenes=case["scenes"], seed=2, lo=case["lo"], hi=case["hi"])
    w.seed = seed
    return w


def _samples(case, seed):
    """Features of the captures' distribution; a sample trains the output of
    the solve it was taken before, the other target is NaN."""
    g = torch.Generator().manual_seed(seed)
    n = case["batch"] * case["steps"]
    u = torch.randn(n, 12, generator=g)
    x = u * torch.tensor(X_STD) + torch.tensor(X_MEAN)
    t = torch.stack([torch.tanh(u[:, 4]) + 0.3 * u[:, 2], 0.5 * u[:, 5] - 0.4 * u[:, 0]], 1)
    t = t + 0.2 * torch.randn(n, 2, generator=g)
    y = t * torch.tensor(Y_STD) + torch.tensor(Y_MEAN)
    which = torch.rand(n, generator=g) < 0.5
    y[which, 0] = math.nan
    y[~which, 1] = math.nan
    return x, y


def _lr(k, steps):
    return 2e-3 * 0.5 * (1.0 + math.cos(math.pi * k / steps))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "passes":
        s["steps"].submit_substeps(s["builder"], s["iters"], s["substeps"], s["first"])
        s["first"] = False
        d = s["data"]
        st = d.read_stats()
        return {"position": d.download(_abi.FE_FIELD_POSITION_A),
                "velocity": d.download(_abi.FE_FIELD_VELOCITY_B),
                "density": d.download(_abi.FE_FIELD_DENSITY),
                "stats": [st.max_speed, st.avg_density_error_f64, st.avg_divergence_error_f64]}
    if kind == "app":
        f = s["frames"]
        st = f.driver.step()
        pos, vel = f.copy_out()
        return {"position": pos, "velocity": vel,
                "stats": [st.max_speed, st.avg_density_error_f64]}
    if kind in ("frames", "batch"):
        f = s["frames"]
        f.sim.step(1, want_stats=False)
        pos, vel = f.copy_out()
        return {"position": pos, "velocity": vel}
    if kind == "sort":
        s["k"].copy_(s["keys"])
        s["v"].copy_(s["vals"])
        lib = s["lib"]
        _abi.check(lib, lib.fe_sort_pairs(
            ctypes.c_void_p(s["k"].data_ptr()), ctypes.c_void_p(s["v"].data_ptr()),
            s["k"].numel(), s["bits"], s["algorithm"],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fe_sort_pairs")
        return {"keys": s["k"], "vals": s["v"]}
    if kind == "water":
        d = s["sim"].data
        lib, h = d._lib, d.handle
        _abi.check(lib, lib.fe_density_splat(h), "fe_density_splat")
        _abi.check(lib, lib.fe_raymarch(h, ctypes.byref(s["cam"])), "fe_raymarch")
        img = s["out"][s["turn"]]
        s["turn"] ^= 1
        t = d.download_async(_abi.FE_FIELD_IMAGE, img.numpy())
        if s["ticket"] is not None:
            d.download_wait(s["ticket"])
        s["ticket"] = t
        return {"image": img}
    m, b, losses = s["model"], s["batch"], []
    for k in range(s["steps"]):
        loss = ctypes.c_float()
        _abi.check(m.lib, m.lib.fe_model_train_step(
            m.handle, ctypes.c_void_p(s["x"].data_ptr() + k * b * 48),
            ctypes.c_void_p(s["y"].data_ptr() + k * b * 8), b, _lr(k, s["steps"]), 1e-5, None,
            ctypes.byref(loss)), "fe_model_train_step")
        losses.append(loss.value)
    return {"parameters": m.parameters(), "losses": losses}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Per particle and pass: positions, velocities and scalars read and
    written once; per neighbour pair some 20 operations in the density pass,
    15 in viscosity and 10 in the sources, the pressure force and its update."""
    kind = case["kind"]
    if kind in ("passes", "app", "frames", "batch"):
        if kind == "batch":
            n = sum(_batch(case, 0).counts)
        else:
            n = case["nx"] * case["ny"] * case["nz"]
        sub = {"passes": case.get("substeps", 1), "app": 4}.get(kind, 1)
        its = 2 * case["iters"] if kind == "passes" else 8
        if case.get("solver") == "tolerance":
            its = 10 if case["cfl"] else 3
        # viscosity, the sources, integrations, search and stats; force + update
        per = 40 + 36 + 60 + 20 + 28 + 36 + 20 + 136 + its * (32 + 44)
        pair = 20 + 15 + 10 + 10 + its * 20
        extra = (1 + (kind == "app")) * 156
        return {"bytes": float(n) * (sub * per + extra),
                "flops": float(n) * PAIRS * sub * pair}
    if kind == "sort":
        # the pairs are copied, read and written
        return {"bytes": 32.0 * case["n"], "flops": 0.0}
    if kind == "water":
        n = case["nx"] * case["ny"] * case["nz"]
        vox, px = case["rx"] * case["ry"] * case["rz"], case["width"] * case["height"]
        return {"bytes": 16.0 * n + 8.0 * vox + 32.0 * px, "flops": 400.0 * vox + 4000.0 * px}
    n = case["batch"] * case["steps"]
    return {"bytes": 56.0 * n, "flops": 6.0 * n * (16 * 64 + 64 * 64 + 2 * 64)}


# ---------------------------------------------------------------------------
# The same passes in 64 bits
# ---------------------------------------------------------------------------
class _Flow:
    """The DFSPH step of one or more scenes laid out back to back, in FP64.
    Only the assignment of particles to cells is decided in FP32, as the step
    defines it (floor(p / h) in single precision)."""

    def __init__(self, scenes, dev):
        """scenes: [(params, positions)] with the same mode, sort and h."""
        self.dev, f64 = dev, torch.float64
        self.p = p = scenes[0][0]
        self.fixed = p.mode == _abi.FE_MODE_FIXED
        self.h, self.m = float(np.float32(p.smoothing_radius)), float(np.float32(p.particle_mass))
        self.rho0, self.omega = float(np.float32(p.target_density)), float(np.float32(p.relax_factor))
        self.dt = float(np.float32(p.dt))
        cnt = [len(x) for _, x in scenes]
        tab = [1 << max(0, (c - 1).bit_length()) for c in cnt]
        sid = torch.repeat_interleave(torch.arange(len(cnt)), torch.tensor(cnt)).to(dev)

        def per(values):
            return torch.tensor(values, device=dev)[sid]

        base = np.concatenate([[0], np.cumsum(tab)[:-1]]).tolist()
        self.table, self.base, self.T = per(tab), per(base), sum(tab)
        self.visc = per([float(np.float32(q.viscosity)) for q, _ in scenes]).to(f64)[:, None]
        self.set_box([q for q, _ in scenes], sid)
        self.xa = torch.cat([torch.as_tensor(x) for _, x in scenes]).to(dev, f64)
        n = self.n = self.xa.shape[0]
        self.va = torch.zeros(n, 3, dtype=f64, device=dev)
        self.pr = torch.zeros(n, dtype=f64, device=dev)
        self.g = torch.tensor([float(np.float32(v)) for v in p.gravity], dtype=f64, device=dev)

    def set_box(self, params, sid=None):
        f64 = torch.float64
        r = torch.tensor([float(np.float32(q.particle_radius)) for q in params])
        lo = torch.tensor([[float(np.float32(v)) for v in q.box_min] for q in params], dtype=f64)
        hi = torch.tensor([[float(np.float32(v)) for v in q.box_max] for q in params], dtype=f64)
        if sid is not None:
            self.sid = sid
        self.lo, self.hi = lo.to(self.dev)[self.sid], hi.to(self.dev)[self.sid]
        self.rad = r.to(self.dev, f64)[self.sid]

    def hash(self, c):
        """c: int64 cell coordinates."""
        k = (c[:, 0] * 73856093) ^ (c[:, 1] * 19349663) ^ (c[:, 2] * 83492791)
        return self.base + ((k & 0xFFFFFFFF) & (self.table - 1))

    def cells(self, x):
        return torch.floor(x.float() / torch.tensor(self.h, dtype=torch.float32, device=self.dev)).long()

    def search(self):
        key = self.hash(self.cells(self.xa))
        if self.p.sort_algorithm == _abi.FE_SORT_BITONIC:
            order = self.bitonic(key)
        else:
            order = torch.sort(key, stable=True).indices
        self.x, self.vb = self.xa[order], self.va[order]
        if self.fixed:
            self.pr = self.pr[order]
        key = key[order]
        cell = self.cells(self.x)
        slots = torch.arange(self.T + 1, device=self.dev)
        first = torch.searchsorted(key, slots)
        gi, gj = [], []
        for z in (-1, 0, 1):
            for y in (-1, 0, 1):
                for x in (-1, 0, 1):
                    k = self.hash(cell + torch.tensor([x, y, z], device=self.dev))
                    a, c = first[k], first[k + 1] - first[k]
                    i = torch.repeat_interleave(torch.arange(self.n, device=self.dev), c)
                    at = torch.arange(i.numel(), device=self.dev) - torch.repeat_interleave(
                        torch.cumsum(c, 0) - c, c)
                    j = a[i] + at
                    near = ((self.x[i] - self.x[j]) ** 2).sum(1) <= self.h * self.h
                    gi.append(i[near])
                    gj.append(j[near])
        i, j = torch.cat(gi), torch.cat(gj)
        rv = self.x[i] - self.x[j]
        r = rv.norm(dim=1)
        q = r / self.h
        k = 8.0 / (math.pi * self.h ** 3)
        w = torch.where(q <= 0.5, k * (6 * q ** 3 - 6 * q ** 2 + 1), k * 2 * (1 - q) ** 3)
        w = torch.where(q >= 1, torch.zeros_like(w), w)
        gf = torch.where(q <= 0.5, k * (18 * q * q - 12 * q), -6 * k * (1 - q) ** 2)
        far = r > 1e-6
        self.rho = self.m * self.total(w, i)
        i, j, w = i[far], j[far], w[far]
        grad = (gf[far] / (self.h * r[far]))[:, None] * rv[far]
        grad[q[far] >= 1] = 0
        self.i, self.j, self.w, self.grad = i, j, w, grad
        mg = self.m * grad
        al = self.total((mg * mg).sum(1), i) + (self.total(mg, i) ** 2).sum(1)
        self.alpha = torch.where(al > 1e-6, al, torch.zeros_like(al))

    def bitonic(self, key):
        n = 1 << max(0, (self.n - 1).bit_length())
        k = torch.full((n,), 1 << 32, dtype=torch.int64, device=self.dev)
        k[: self.n] = key
        v = torch.arange(n, device=self.dev)
        h = 2
        while h <= n:
            step = h // 2
            while step:
                t = torch.arange(n // 2, device=self.dev)
                a = (t // step) * step * 2 + t % step
                b = a + step
                up = (a & h) == 0
                swap = torch.where(up, k[a] > k[b], k[a] < k[b])
                a, b = a[swap], b[swap]
                k[a], k[b] = k[b], k[a]
                v[a], v[b] = v[b], v[a]
                step //= 2
            h *= 2
        return v[: self.n]

    def total(self, t, i):
        return torch.zeros((self.n,) + t.shape[1:], dtype=t.dtype, device=self.dev).index_add_(0, i, t)

    def divergence(self, v):
        return self.m * self.total(((v[self.i] - v[self.j]) * self.grad).sum(1), self.i)

    def solve(self, density):
        p, dt = self.p, self.dt
        tol = p.solver == _abi.FE_SOLVER_TOLERANCE
        most = p.max_iterations if tol else (p.density_solver_iterations if density
                                             else p.divergence_solver_iterations)
        for it in range(most):
            pr = self.pr / (self.rho * self.rho)
            acc = -self.total((self.m * (pr[self.i] + pr[self.j]))[:, None] * self.grad, self.i)
            self.acc = acc
            err = self.src - dt * self.divergence(acc)
            aii = -(dt / (self.rho * self.rho)) * self.alpha
            acts = (self.alpha > 1e-6) & (aii.abs() > 1e-20)
            new = self.pr + self.omega * err / torch.where(acts, aii, torch.ones_like(aii))
            e = torch.where(new > 0, err.abs(), self.pr * aii.abs() / self.omega)
            e = torch.where(acts, e, torch.zeros_like(e))
            self.pr = torch.where(acts, new.clamp_min(0), self.pr)
            limit = p.density_tolerance if density else p.divergence_tolerance
            if tol and it + 1 >= p.min_iterations and float((dt * e).mean()) / self.rho0 <= limit:
                break

    def substep(self):
        dt = self.dt
        i, j, v = self.i, self.j, self.vb
        s = self.total((self.m / self.rho[j] * self.w)[:, None] * (v[j] - v[i]), i)
        self.va = v + self.visc * s + self.g * dt
        self.src = (self.rho0 - self.rho) / dt - self.divergence(self.va)
        self.pr = torch.zeros_like(self.pr)
        self.solve(True)
        v = self.va + self.acc * dt
        x = self.x + v * dt
        for a in (1, 0, 2):
            lo, hi, r = self.lo[:, a], self.hi[:, a], self.rad
            below, above = x[:, a] < lo + r, x[:, a] > hi - r
            x[:, a] = torch.where(below, lo + r + 0.001, torch.where(above, hi - r - 0.001, x[:, a]))
            hit = (below | above)[:, None]
            f = torch.full((3,), 0.95, dtype=v.dtype, device=self.dev)
            f[a] = -0.5
            v = torch.where(hit, v * f, v)
        self.xa, self.va = x, v
        self.search()
        v = self.vb if self.fixed else self.va
        self.src = -self.divergence(v)
        self.solve(False)
        v = v + self.acc * dt
        if self.fixed:
            self.vb = v
        else:
            self.va = v
        return v

    def out(self):
        one, zero = torch.ones(self.n, 1).to(self.xa), torch.zeros(self.n, 1).to(self.xa)
        return {"position": torch.cat([self.xa, one], 1), "velocity": torch.cat([self.vb, zero], 1)}

    def stats(self, v):
        return [float(v.norm(dim=1).max()), float((self.rho - self.rho0).abs().mean()),
                float(self.src.abs().mean())]


def exact(case, seed):
    kind, cuda = case["kind"], torch.cuda.is_available()
    dev = torch.device("cuda" if cuda else "cpu")
    if kind == "train":
        return _train64(case, seed)
    # sorts are whole numbers; the water pass decides hits at the grid's
    # resolution, and the network's start is rounded to 16 bits on its way
    if kind in ("sort", "water") or case.get("learned") or case.get("cfl", 0.0):
        return None
    if kind == "batch":
        w = _batch(case, seed)
        scenes = list(zip(w.params(), w.positions()))
    else:
        p, pos = (_dam if kind == "frames" else _app)(case, seed)
        if kind == "passes" and case["sort"] == "bitonic":
            p.sort_algorithm = _abi.FE_SORT_BITONIC
        scenes = [(p, pos)]
    n = sum(len(x) for _, x in scenes)
    steps = {"passes": case.get("substeps", 0), "app": 8}.get(kind, case.get("warm", 0) + 1)
    if n * steps > (12_000_000 if cuda else 150_000):
        return None
    if kind == "passes":
        scenes[0][0].density_solver_iterations = case["iters"]
        scenes[0][0].divergence_solver_iterations = case["iters"]
    f = _Flow(scenes, dev)
    if kind == "app":
        p = scenes[0][0]
        box = frame.CollisionBox(list(p.box_min), list(p.box_max), 0.3, 0.5)
        for _ in range(2):
            q = _abi.copy_params(p)
            q.box_min[:] = [float(v) for v in box.min]
            f.set_box([q])
            box.update(1.0 / 60.0)
            f.search()
            for _ in range(4):
                v = f.substep()
        return {**f.out(), "stats": f.stats(v)[:2]}
    f.search()
    for _ in range(steps):
        v = f.substep()
    if kind == "passes":
        return {**f.out(), "density": f.rho, "stats": f.stats(v)}
    return f.out()


def _train64(case, seed):
    f64 = torch.float64
    x, y = _samples(case, seed)
    x = (x.to(f64) - torch.tensor(X_MEAN, dtype=f64)) / torch.tensor(X_STD, dtype=f64)
    y = (y.to(f64) - torch.tensor(Y_MEAN, dtype=f64)) / torch.tensor(Y_STD, dtype=f64)
    x = torch.cat([x, torch.zeros(x.shape[0], 4, dtype=f64)], 1)
    p = torch.from_numpy(_network(seed)).to(f64).requires_grad_(True)
    m, v, losses, b = torch.zeros_like(p), torch.zeros_like(p), [], case["batch"]
    for k in range(case["steps"]):
        w1, w2, w3, b1, b2, b3 = torch.split(p, [1024, 4096, 128, 64, 64, 2])
        a = torch.nn.functional.silu(x[k * b:(k + 1) * b] @ w1.view(64, 16).T + b1)
        a = torch.nn.functional.silu(a @ w2.view(64, 64).T + b2)
        e = a @ w3.view(2, 64).T + b3 - y[k * b:(k + 1) * b]
        loss = torch.where(torch.isnan(e), torch.zeros_like(e), e).square().sum() / b
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            g = g + 1e-5 * p
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            step = (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
            p = (p - _lr(k, case["steps"]) * step).requires_grad_(True)
        losses.append(float(loss))
    return {"parameters": p.detach(), "losses": losses}
