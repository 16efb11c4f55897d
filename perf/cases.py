"""The work that programs built on this package have it do, as cases to be timed.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more
of the same ranges, `prepare(case, seed)` what a program holds before the call (inputs,
solvers, scratch), `run(state)` one pass through the public entry points, `work(case)`
the bytes and operations that pass cannot do without, `exact(case, seed)` the same
outputs in 64 bits where plain torch arithmetic gives them.
"""
from __future__ import annotations

import numpy as np
import torch

from inchman_b200 import _lib
from inchman_b200 import ensemble as ens
from inchman_b200 import gray_scott as gs
from inchman_b200 import individual as ind
from inchman_b200.model import DiffusionModel, lotka_volterra_model
from inchman_b200.solver import Solver

DEV = "cuda"
THETA = (0.04, 0.06, 0.16, 0.08)      # F, k, Du, Dv of the Gray-Scott workload


def listed():
    return [
        # One deterministic solve to the end time: the benchmark's lattice and length.
        {"name": "gs_forward_256", "kind": "gs_forward", "n": 256, "steps": 10000, "drift": False},
        # A parameter scan: many lattices with their own rates, solved side by side.
        {"name": "gs_batch_64x128", "kind": "gs_batch", "n": 128, "steps": 2000, "batch": 64},
        # One iteration of a parameter fit: forward with checkpoints, then the adjoint.
        {"name": "gs_gradient_256", "kind": "gs_gradient", "n": 256, "steps": 2000, "f64": False, "drift": False},
        # The same in double precision with advection, where the gradient is checked
        # against finite differences.
        {"name": "gs_gradient_128_f64", "kind": "gs_gradient", "n": 128, "steps": 1000, "f64": True, "drift": True},
        # A heterogeneous ensemble: every instance its own grid, network and rates.
        {"name": "ensemble_random_592", "kind": "ensemble_random", "instances": 592, "max_time": 0.1},
        # A handful of realisations of one small model run to its end time (A + B <-> C).
        {"name": "ensemble_32x32_x16", "kind": "ensemble_replicas", "width": 32, "instances": 16, "max_time": 2.0},
        # A program's own event loop around the wide solver: reaction window, then jumps.
        {"name": "jumps_128x128_x64", "kind": "jumps", "width": 128, "height": 128, "realisations": 64, "events": 16},
        # The same loop with drift-diffusion sweeps on per-cell fields (predator and prey).
        {"name": "drift_512x512_x32", "kind": "drift", "width": 512, "realisations": 32, "events": 8},
        # Brownian particles that annihilate in pairs: set up, run one output interval,
        # read back.
        {"name": "particles_2p22_1024", "kind": "particles", "n": 1 << 22, "grid": 1024, "steps": 100},
        # The list primitives at the size where they stream from memory.
        {"name": "scan_2p27", "kind": "scan", "n": 1 << 27},
        {"name": "sort_2p24_32bit", "kind": "sort", "n": 1 << 24, "bits": 32},
        # The smallest calls: sort a short list by cell, index it, bring it to new counts.
        {"name": "upkeep_32x32", "kind": "upkeep", "width": 32, "mean": 4.0},
    ]


def _log_int(rng, lo, hi):
    """An integer whose logarithm is uniform over [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("gs_forward", "gs_batch", "gs_gradient", "ensemble_random", "ensemble_replicas", "jumps",
                       "drift", "particles", "scan", "sort", "upkeep"))
    if kind == "gs_forward":
        # lattice sides the solver accepts, the ones without a kernel of their own among them
        n = rng.choice((64, 75, 96, 100, 128, 160, 192, 256, 256, 320, 416))
        top = min(10000, int(10000 * (256 / n) ** 2))
        return {"kind": kind, "n": n, "steps": _log_int(rng, 300, top), "drift": rng.random() < 0.3}
    if kind == "gs_batch":
        n = rng.choice((64, 128, 256))
        return {"kind": kind, "n": n, "steps": _log_int(rng, 200, 2000 if n < 256 else 1000),
                "batch": _log_int(rng, 2, 64 if n > 64 else 256) if n < 256 else _log_int(rng, 2, 24)}
    if kind == "gs_gradient":
        f64 = rng.random() < 0.4
        n = rng.choice((64, 96, 128) if f64 else (64, 96, 128, 192, 256, 256))
        return {"kind": kind, "n": n, "steps": _log_int(rng, 150, 1000 if f64 else 2000), "f64": f64,
                "drift": rng.random() < 0.5}
    if kind == "ensemble_random":
        return {"kind": kind, "instances": _log_int(rng, 40, 592), "max_time": round(0.02 + 0.08 * rng.random(), 3)}
    if kind == "ensemble_replicas":
        w = rng.randint(16, 64)
        return {"kind": kind, "width": w, "instances": _log_int(rng, 2, 64),
                "max_time": round(0.5 + 1.5 * rng.random(), 3)}
    if kind == "jumps":
        w, h = rng.randint(24, 256), rng.randint(24, 256)
        return {"kind": kind, "width": w, "height": h, "events": rng.randint(4, 16),
                "realisations": _log_int(rng, 1, max(1, min(256, (1 << 20) // (w * h))))}
    if kind == "drift":
        w = rng.randint(48, 512)
        return {"kind": kind, "width": w, "events": rng.randint(2, 8),
                "realisations": _log_int(rng, 1, max(1, min(256, 32 * 512 * 512 // (w * w))))}
    if kind == "particles":
        grid = _log_int(rng, 64, 1024)
        return {"kind": kind, "n": _log_int(rng, grid * grid // 4, min(1 << 22, 8 * grid * grid)), "grid": grid,
                "steps": rng.randint(20, 100)}
    if kind == "scan":
        return {"kind": kind, "n": _log_int(rng, 100, 1 << 27)}
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 100, 1 << 24), "bits": rng.randint(8, 32)}
    return {"kind": kind, "width": _log_int(rng, 24, 1024), "mean": round(1.0 + 7.0 * rng.random(), 2)}


# -- Gray-Scott ---------------------------------------------------------------------

def _gs_inputs(case, seed):
    dtype = np.float64 if case.get("f64") else np.float32
    cfg = gs.GrayScottConfig(n=case["n"], steps=case["steps"], seed=seed)
    if case.get("drift"):
        cfg.vx, cfg.vy = 0.05, -0.03
    u0, v0 = cfg.initial_state(dtype)
    return cfg, torch.from_numpy(u0).to(DEV), torch.from_numpy(v0).to(DEV)


def _gs_batch_inputs(case, seed):
    cfg, u0, v0 = _gs_inputs(case, seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    shape = (case["batch"],) + tuple(u0.shape)
    u = u0 + 0.005 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float32)
    v = v0 + 0.005 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float32)
    rng = np.random.default_rng(seed)
    th = np.tile(np.array(THETA + (0.0, 0.0)), (case["batch"], 1))
    th[:, 0] *= rng.uniform(0.95, 1.05, case["batch"])
    th[:, 1] *= rng.uniform(0.97, 1.03, case["batch"])
    return cfg, u.contiguous(), v.contiguous(), th


def _gs_upstream(case, seed, like):
    """Gradients of a loss with respect to the final state, as a fit would pass them."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1)
    return [torch.randn(like.shape, generator=g, device=DEV, dtype=like.dtype) for _ in range(2)]


def _lap(a):
    return (torch.roll(a, 1, -1) + torch.roll(a, -1, -1) + torch.roll(a, 1, -2) + torch.roll(a, -1, -2)) - 4 * a


def _gs_step(u, v, th, dt):
    F, k, Du, Dv, vx, vy = th
    r = u * v * v
    un = u + dt * (Du * _lap(u) - r + F * (1 - u))
    vn = v + dt * (Dv * _lap(v) + r - (F + k) * v)
    if vx is not None:
        un = un - dt * 0.5 * (vx * (torch.roll(u, -1, -1) - torch.roll(u, 1, -1))
                              + vy * (torch.roll(u, -1, -2) - torch.roll(u, 1, -2)))
        vn = vn - dt * 0.5 * (vx * (torch.roll(v, -1, -1) - torch.roll(v, 1, -1))
                              + vy * (torch.roll(v, -1, -2) - torch.roll(v, 1, -2)))
    return un, vn


def _gs_exact_forward(case, seed):
    if case["kind"] == "gs_batch":
        cfg, u, v, th = _gs_batch_inputs(case, seed)
        # the rates reach the kernels as float32 numbers
        t = torch.from_numpy(th.astype(np.float32).astype(np.float64)).to(DEV)[:, :, None, None]
        par = [t[:, 0], t[:, 1], t[:, 2], t[:, 3], None, None]
    else:
        cfg, u, v = _gs_inputs(case, seed)
        par = [float(np.float32(x)) for x in cfg.theta()]
        if not case["drift"]:
            par[4] = par[5] = None
    u, v = u.double(), v.double()
    for _ in range(case["steps"]):
        u, v = _gs_step(u, v, par, cfg.dt)
    return u, v


def _gs_exact_gradient(case, seed):
    cfg, u, v = _gs_inputs(case, seed)
    lu, lv = (x.double() for x in _gs_upstream(case, seed, u))
    u, v = u.double(), v.double()
    cast = float if case["f64"] else (lambda x: float(np.float32(x)))
    F, k, Du, Dv, vx, vy = (cast(x) for x in cfg.theta())
    us, vs = [], []
    for _ in range(case["steps"]):
        us.append(u)
        vs.append(v)
        u, v = _gs_step(u, v, (F, k, Du, Dv, vx, vy), cfg.dt)
    gth = torch.zeros(6, dtype=torch.float64, device=DEV)
    dx = lambda a: torch.roll(a, -1, -1) - torch.roll(a, 1, -1)      # noqa: E731
    dy = lambda a: torch.roll(a, -1, -2) - torch.roll(a, 1, -2)      # noqa: E731
    dt = cfg.dt
    for j in range(case["steps"] - 1, -1, -1):
        a, b = us[j], vs[j]
        gth += dt * torch.stack([(lu * (1 - a)).sum() - (lv * b).sum(), -(lv * b).sum(), (lu * _lap(a)).sum(),
                                 (lv * _lap(b)).sum(), -0.5 * ((lu * dx(a)).sum() + (lv * dx(b)).sum()),
                                 -0.5 * ((lu * dy(a)).sum() + (lv * dy(b)).sum())])
        d = lv - lu
        nu = lu + dt * (Du * _lap(lu) + b * b * d - F * lu + 0.5 * (vx * dx(lu) + vy * dy(lu)))
        nv = lv + dt * (Dv * _lap(lv) + 2 * a * b * d - (F + k) * lv + 0.5 * (vx * dx(lv) + vy * dy(lv)))
        lu, lv = nu, nv
    return u, v, lu, lv, gth


# -- stochastic models ----------------------------------------------------------------

def _abc_model(width, height, max_time):
    """A + B <-> C with D = (1, 1, 0.5) on unit cells, reflecting walls."""
    m = DiffusionModel(width=width, height=height, physical_length=float(width), p0=0.1, max_time=max_time,
                       output_interval=1.0, solver=_lib.STOCHASTIC_HOMOGENEOUS)
    m.add_species("A", 1.0, 100.0).add_species("B", 1.0, 100.0).add_species("C", 0.5, 0.0)
    m.add_reaction("bind", {"A": 1, "B": 1}, {"C": 1}, 0.01)
    m.add_reaction("unbind", {"C": 1}, {"A": 1, "B": 1}, 0.1)
    return m


class _DeviceArray:
    """The solver's state in device memory, for torch to read without a copy."""

    def __init__(self, solver):
        self.__cuda_array_interface__ = {"shape": solver.shape, "typestr": "<i4", "version": 2,
                                         "data": (solver.device_state_ptr(), False), "strides": None}


def _run_events(st):
    """`events` passes of the event loop from a fresh initial state: the reaction window
    up to the next diffusion time, then the species that are due."""
    s = st["solver"]
    s.init_poisson(st["lam"])
    t = st["t"]
    for e in range(st["events"]):
        due = s.get_next_diffusion_time()
        now = due.min()
        seed = s.do_reactions(float(now - t), 64 * e)
        for i in range(due.size):
            if due[i] <= now:
                seed = s.diffuse(i, float(now), seed)
        t = now
    st["t"] = t
    return torch.as_tensor(_DeviceArray(s), device=DEV).clone()


# -- preparation ------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    if kind == "gs_forward":
        cfg, u0, v0 = _gs_inputs(case, seed)
        return {"kind": kind, "u0": u0, "v0": v0, "p": cfg.params()}
    if kind == "gs_batch":
        cfg, u0, v0, th = _gs_batch_inputs(case, seed)
        return {"kind": kind, "u0": u0, "v0": v0, "theta": th, "p": cfg.params()}
    if kind == "gs_gradient":
        cfg, u0, v0 = _gs_inputs(case, seed)
        th = torch.tensor(cfg.theta(), dtype=torch.float64, device=DEV).requires_grad_()
        return {"kind": kind, "u0": u0.requires_grad_(), "v0": v0.requires_grad_(), "theta": th, "dt": cfg.dt,
                "steps": cfg.steps, "up": _gs_upstream(case, seed, u0), "fn": gs.GrayScott()}
    if kind in ("ensemble_random", "ensemble_replicas"):
        if kind == "ensemble_random":
            # the networks of one study, its realisations seeded anew
            specs = ens.random_ensemble(case["instances"], 2024, max_time=case["max_time"])
            for i, sp in enumerate(specs):
                sp.seed = (seed * 7919 + i) & 0xFFFFFFFF
        else:
            m = _abc_model(case["width"], case["width"], case["max_time"])
            specs = ens.replicate(m, [100.0, 100.0, 0.0], case["instances"], seed)
        e = ens.Ensemble(specs)
        e.configure(1024, 1)          # the shape the package's own ensemble program runs
        return {"kind": kind, "ens": e, "state": e.alloc_state()}
    if kind == "jumps":
        m = _abc_model(case["width"], case["height"], 1e6)
        return {"kind": kind, "solver": Solver(m, realisations=case["realisations"], seed=seed),
                "lam": [100.0, 100.0, 0.0], "t": np.float32(0), "events": case["events"]}
    if kind == "drift":
        m = lotka_volterra_model(width=case["width"], max_time=1e6, seed=seed)
        return {"kind": kind, "solver": Solver(m, realisations=case["realisations"], seed=seed),
                "lam": [50.0, 50.0], "t": np.float32(0), "events": case["events"]}
    if kind == "particles":
        x, y, sp = ind.uniform_particles(case["n"], case["grid"], seed)
        p = ind.Particles(case["n"], case["grid"], D=0.5, vx=0.1, vy=0.0, dt=1.0, p_react=0.005, seed=seed)
        frame = (np.zeros(case["n"], np.float32), np.zeros(case["n"], np.float32), np.zeros(case["n"], np.uint8))
        return {"kind": kind, "p": p, "x": x, "y": y, "sp": sp, "steps": case["steps"], "frame": frame}
    n = case.get("n")
    if kind == "scan":
        x = torch.randint(0, 16, (n,), dtype=torch.int32, device=DEV, generator=g)
        return {"kind": kind, "x": x, "scratch": ind.scan_scratch(n)}
    if kind == "sort":
        b = case["bits"]
        k = torch.randint(0, 1 << b, (n,), dtype=torch.int64, device=DEV, generator=g).to(torch.int32)
        return {"kind": kind, "keys": k, "vals": torch.arange(n, dtype=torch.int32, device=DEV), "bits": b,
                "scratch": ind.sort_scratch(n, b)}
    # upkeep: an unsorted list of individuals after a move, the counts the reactions want
    cells = case["width"] ** 2
    n = int(case["mean"] * cells)
    npool = cells + n // 4
    keys = torch.randint(0, cells, (n,), dtype=torch.int32, device=DEV, generator=g)
    perm = torch.randperm(n + npool, dtype=torch.int32, device=DEV, generator=g)
    # a third of the individuals vanish and as many appear elsewhere
    moved = torch.where(torch.rand(n, generator=g, device=DEV) < 0.33,
                        torch.randint(0, cells, (n,), dtype=torch.int32, device=DEV, generator=g), keys)
    goal = torch.bincount(moved, minlength=cells).to(torch.int32)
    bits = max(1, (cells - 1).bit_length())
    return {"kind": "upkeep", "keys": keys, "ids": perm[:n].contiguous(), "pool": perm[n:].contiguous(), "goal": goal,
            "cells": cells, "bits": bits, "seed": seed, "sort": ind.sort_scratch(n, bits),
            "scan": ind.scan_scratch(cells)}


def run(st):
    kind = st["kind"]
    if kind == "gs_forward":
        return gs.forward(st["u0"], st["v0"], st["p"])
    if kind == "gs_batch":
        return gs.forward_batch(st["u0"], st["v0"], st["p"], st["theta"])
    if kind == "gs_gradient":
        u, v = st["fn"].apply(st["u0"], st["v0"], st["theta"], st["steps"], st["dt"], 0)
        gu, gv, gt = torch.autograd.grad((u, v), (st["u0"], st["v0"], st["theta"]), st["up"])
        return u.detach(), v.detach(), gu, gv, gt
    if kind in ("ensemble_random", "ensemble_replicas"):
        st["ens"].init_poisson(st["state"])
        st["ens"].run(st["state"])
        return st["state"]
    if kind in ("jumps", "drift"):
        return _run_events(st)
    if kind == "particles":
        p = st["p"]
        p.set(st["x"], st["y"], st["sp"])
        p.step(st["steps"])
        # a frame of fixed size for the output file, empty slots zero
        for slot, values in zip(st["frame"], p.get()):
            slot[:values.size] = values
            slot[values.size:] = 0
        return st["frame"]
    if kind == "scan":
        return ind.exclusive_scan_u32(st["x"], st["scratch"])
    if kind == "sort":
        return ind.sort_pairs_u32(st["keys"], st["vals"], st["bits"], st["scratch"])[:2]
    keys, ids, _ = ind.sort_pairs_u32(st["keys"], st["ids"], st["bits"], st["sort"])
    start, count = ind.cell_offsets(keys, st["cells"], st["scan"])
    new = ind.maintain_population(keys, ids, start, count, st["goal"], st["pool"], st["seed"], 1)
    return (keys, ids, start, count) + tuple(new)


def work(case):
    kind = case["kind"]
    if kind == "gs_forward":
        cells = case["n"] ** 2
        return {"bytes": 16.0 * cells, "flops": (29.0 if case["drift"] else 25.0) * cells * case["steps"]}
    if kind == "gs_batch":
        cells = case["n"] ** 2 * case["batch"]
        return {"bytes": 16.0 * cells, "flops": 25.0 * cells * case["steps"]}
    if kind == "gs_gradient":
        # a forward step, and a transposed step with the six parameter sums
        cells, e = case["n"] ** 2, 8 if case["f64"] else 4
        return {"bytes": 8.0 * e * cells, "flops": (25.0 + 43.0) * cells * case["steps"]}
    # one random block (ten rounds, about 60 operations) per cell, species and event is
    # the least that the samplers need
    if kind == "ensemble_random":
        # the ensemble's means: 5,800 cells, 8 species, one jump per species each 1 / (60 D)
        cells, events = 5800.0 * case["instances"], 65.0 * case["max_time"]
        return {"bytes": 8.0 * 8 * cells, "flops": 60.0 * 8 * cells * events}
    if kind == "ensemble_replicas":
        cells = case["width"] ** 2 * case["instances"]
        return {"bytes": 8.0 * 3 * cells, "flops": 60.0 * 3.5 * cells * 60.0 * case["max_time"]}
    if kind == "jumps":
        cells = case["width"] * case["height"] * case["realisations"]
        return {"bytes": 8.0 * 3 * cells, "flops": 60.0 * 3.5 * cells * case["events"]}
    if kind == "drift":
        cells = case["width"] ** 2 * case["realisations"]
        return {"bytes": 8.0 * 2 * cells, "flops": 60.0 * 3.0 * cells * case["events"]}
    if kind == "particles":
        # each step reads and writes every particle once
        return {"bytes": 18.0 * case["n"] * case["steps"], "flops": 100.0 * case["n"] * case["steps"]}
    if kind == "scan":
        return {"bytes": 8.0 * case["n"], "flops": float(case["n"])}
    if kind == "sort":
        return {"bytes": 16.0 * case["n"], "flops": 0.0}
    cells = case["width"] ** 2
    n = case["mean"] * cells
    return {"bytes": 16.0 * n + 16.0 * n + 24.0 * cells + 8.0 * (cells + n / 4), "flops": 0.0}


def exact(case, seed):
    if case["kind"] in ("gs_forward", "gs_batch"):
        return _gs_exact_forward(case, seed)
    if case["kind"] == "gs_gradient":
        return _gs_exact_gradient(case, seed)
    return None          # counts and sorted lists are whole numbers; particle moves are random draws
