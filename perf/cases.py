"""The workloads whose speed this framework is judged by: what a user's program has it do, through
its public entry points, from single coupled steps on a small mesh to the 4M-cell solve.

A case is a dict of plain values; ``prepare`` builds the model, network or batch a program keeps in
hand, ``run`` makes one pass, ``work`` says what a pass cannot do without and ``exact`` restates the
single- and dual-porosity step and the network's training step in plain torch, in 64 bits.

Meshes are seeded constructions of ``workloads``; the seed of a state moves the initial flow, the
porosity and the friction.  Host tables of a construction are kept between states of one process.
"""
from __future__ import annotations

import copy
import functools
import importlib
import math

import numpy as np
import torch

sw2d = importlib.import_module("inria-internship-project-sw2d-enzyme_b200")

GRAVITY, SMALL = 9.81, 1e-16


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # one step per call, the state read back into host arrays: a model coupled step by step to
        # another program (a drainage network, a rainfall model) on a small mesh
        {"name": "sp_coupled_2k", "kind": "forward", "flow": "dam", "scheme": "muscl_evr", "cells": 2000, "steps": 1,
         "host": True},
        # the size and options of the reference's shipped flume case: Godunov, blending topography,
        # anisotropic Strickler friction, head loss, an inflow hydrograph
        {"name": "sp_flume_5k", "kind": "forward", "flow": "channel", "scheme": "godunov", "cells": 4800, "steps": 64,
         "host": False},
        # the dam break on a randomly numbered Delaunay mesh
        {"name": "sp_dam_20k", "kind": "forward", "flow": "delaunay", "scheme": "muscl_evr", "cells": 20000, "steps": 64,
         "host": False},
        # moving flow with wet/dry fronts over Gaussian bumps, a mesh of ordinary size
        {"name": "sp_bumps_250k", "kind": "forward", "flow": "bumps", "scheme": "muscl_evr", "cells": 250000, "steps": 32,
         "host": False},
        # the benchmark's large solve: a lake at rest between dry bumps
        {"name": "sp_lake_4m", "kind": "forward", "flow": "lake", "scheme": "muscl_evr", "cells": 4000000, "steps": 16,
         "host": False},
        # dual integral porosity with momentum dissipation
        {"name": "dip_300k", "kind": "forward", "flow": "dip", "scheme": "muscl_evr", "cells": 300000, "steps": 16,
         "host": False},
        # depth-dependent porosity
        {"name": "ddp_200k", "kind": "forward", "flow": "ddp", "scheme": "godunov", "cells": 200000, "steps": 16,
         "host": False},
        # one gradient of a 4D-Var iteration: new friction, the reverse sweep over a recorded run
        {"name": "adjoint_100k", "kind": "adjoint", "cells": 100000, "steps": 100, "every": 25},
        # one iteration of the porosity assimilation: dry run, replayed cost and gradient
        {"name": "porosity_10k", "kind": "porosity", "cells": 10000, "steps": 100, "every": 30},
        # an ensemble of uneven meshes (perturbed friction), restarted from its saved points
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "low": 2000, "high": 60000, "steps": 32},
        # the learned closure in the cell update of the dual integral porosity model
        {"name": "closure_500k", "kind": "closure", "cells": 500000, "steps": 8},
        # one training step of the closure's network on a mini-batch of the default size
        {"name": "mlp_step_4096", "kind": "mlp", "batch": 4096},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["forward"] * 7 + ["adjoint", "porosity", "ensemble", "closure", "mlp"])
    if kind == "forward":
        flow = rng.choice(["dam", "channel", "delaunay", "bumps", "lake", "dip", "ddp"])
        high = {"delaunay": 60000, "ddp": 300000}.get(flow, 1000000)
        scheme = "godunov" if flow == "ddp" else rng.choice(["muscl_evr", "godunov"])
        return {"kind": kind, "flow": flow, "scheme": scheme, "cells": _log_int(rng, 500, high),
                "steps": _log_int(rng, 1, 64), "host": rng.random() < 0.3}
    if kind == "adjoint":
        return {"kind": kind, "cells": _log_int(rng, 2000, 300000), "steps": _log_int(rng, 20, 120),
                "every": rng.randint(7, 40)}
    if kind == "porosity":
        return {"kind": kind, "cells": _log_int(rng, 1000, 60000), "steps": _log_int(rng, 20, 120),
                "every": rng.randint(7, 40)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 40), "low": _log_int(rng, 500, 3000),
                "high": _log_int(rng, 5000, 80000), "steps": _log_int(rng, 4, 64)}
    if kind == "closure":
        return {"kind": kind, "cells": _log_int(rng, 2000, 800000), "steps": _log_int(rng, 1, 32)}
    return {"kind": kind, "batch": _log_int(rng, 100, 100000)}


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _construction(flow, scheme, cells, mesh_seed=1):
    """The seeded construction (mesh and maps) a case stands on; host tables, read only."""
    w = sw2d.workloads
    if flow == "dam":
        return w.dam_break(n_cells=cells, scheme=scheme, seed_mesh=mesh_seed)
    if flow == "delaunay":
        return w.dam_break(n_cells=cells, scheme=scheme, mesh="delaunay", seed_mesh=mesh_seed)
    if flow == "unfrictioned":
        return w.dam_break(n_cells=cells, scheme=scheme, friction="none", seed_mesh=mesh_seed)
    if flow == "bumps":
        return w.gaussian_bumps(n_cells=cells, scheme=scheme, initial="dam", seed_mesh=mesh_seed)
    if flow == "lake":
        return w.gaussian_bumps(n_cells=cells, scheme=scheme, initial="lake", seed_mesh=mesh_seed)
    if flow == "channel":
        topo = "blending" if scheme == "godunov" else "discontinuous"
        return w.channel_features(n_cells=cells, scheme=scheme, topo=topo, t_max=1.0e6)
    if flow == "dip":
        return w.dip_channel(n_cells=cells, scheme=scheme, t_max=1.0e6)
    if flow == "ddp":
        return w.ddp_channel(n_cells=cells, laws="linear", moving=True, t_max=1.0e6)
    raise ValueError(flow)


def _inputs(flow, scheme, cells, seed, mesh_seed=1):
    """The construction with this seed's initial flow, porosity and friction, and its start time."""
    base = _construction(flow, scheme, cells, mesh_seed)
    c = copy.copy(base)
    m = base.mesh
    rng = np.random.default_rng(int(seed))
    a = rng.uniform(0.0, 2.0 * np.pi, 4)
    span_x, span_y = max(np.ptp(m.cell_x), 1e-9), max(np.ptp(m.cell_y), 1e-9)
    wave = (np.sin(2 * np.pi * (m.cell_x - m.cell_x.min()) / span_x + a[0]) *
            np.cos(2 * np.pi * (m.cell_y - m.cell_y.min()) / span_y + a[1]))
    side = np.cos(4 * np.pi * (m.cell_x - m.cell_x.min()) / span_x + a[2])
    if flow == "lake":  # at rest: the free surface is flat, at a level of its own
        level = 2.0 + rng.uniform(-0.05, 0.05)
        c.h0 = np.maximum(level - m.cell_z_b, 0.0)
    elif flow == "ddp":
        c.h0 = base.h0 * (1.0 + 0.05 * wave)
        c.q0, c.r0 = base.q0 * (1.0 + 0.3 * side), base.r0 * (1.0 + 0.3 * wave)
    else:  # a moving flow, up to a few tenths of the wave speed
        c.h0 = base.h0 * (1.0 + 0.05 * wave)
        speed = np.sqrt(GRAVITY * c.h0)
        c.q0, c.r0 = 0.3 * c.h0 * speed * side, 0.2 * c.h0 * speed * wave
    if base.friction is not None:
        f = 1.0 + 0.2 * rng.uniform(-1.0, 1.0, m.cell_nb)
        c.friction = np.stack([base.friction[0] * f, base.friction[1] * f, base.friction[2]])
    if flow in ("dam", "delaunay", "unfrictioned"):
        c.phi = np.clip(base.phi + 0.02 * wave, 0.05, 1.0)
    # the hydrographs of the channels carry their flow from a few seconds on
    return c, (8.0 if flow in ("channel", "dip", "ddp") else 0.0)


def _model(flow, scheme, cells, seed, mesh_seed=1):
    case, t0 = _inputs(flow, scheme, cells, seed, mesh_seed)
    model = sw2d.SpModel(case)
    if t0:
        model.set_time(t0, 0.0)
    return model, case


def _forward_state(model, case, steps, host):
    s = {"model": model, "steps": steps, "host": host, "n": model.n}
    if case.is_ddp:  # restarted from the caller's own arrays: the model's state and its time
        s["start"] = [torch.from_numpy(v).cuda() for v in model.state()]
        s["time"] = model.time
    else:
        model.save_point()
    if not host:
        s["out"] = torch.empty((3, model.n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    model.prepare()
    return s


def _network(seed, scale):
    """A network with random weights whose outputs are multiplied by `scale`."""
    norm = np.concatenate([np.zeros(10), np.ones(10), np.zeros(2), np.full(2, scale)]).astype(np.float32)
    return sw2d.closure.MLP(sw2d.closure.init_params(int(seed)), norm)


def _batch_inputs(batch, seed):
    rng = np.random.default_rng(int(seed))
    x = rng.normal(size=(batch, 10)).astype(np.float32)
    t = np.stack([np.sin(x[:, 0]) * x[:, 1], 0.5 * x[:, 2] - np.tanh(x[:, 3])], 1).astype(np.float32)
    return x, t + 0.1 * rng.normal(size=t.shape).astype(np.float32)


@functools.lru_cache(maxsize=16)
def _step_length(cells):
    """Length of an early time step of the frictionless dam break, for the assimilation window."""
    probe = sw2d.SpModel(_construction("unfrictioned", "muscl_evr", cells))
    probe.step(3)
    dt = probe.dt
    probe.close()
    return dt


def _member_sizes(case):
    k = max(1, case["members"] - 1)
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [int(round(math.exp(lo + (hi - lo) * i / k))) for i in range(case["members"])]


def _member_flow(i):
    return "dam" if i % 2 == 0 else "bumps"


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forward":
        model, c = _model(case["flow"], case["scheme"], case["cells"], seed)
        return {"kind": kind, **_forward_state(model, c, case["steps"], case["host"])}
    if kind == "closure":
        model, c = _model("dip", "godunov", case["cells"], seed)
        net = _network(seed, 1e-6)  # corrections small against the discharges
        model.set_closure(net, np.full(10, -1e30, np.float32), np.full(10, 1e30, np.float32))
        return {"kind": "forward", "net": net, **_forward_state(model, c, case["steps"], False)}
    if kind == "adjoint":
        model, c = _model("dam", "muscl_evr", case["cells"], seed)
        rng = np.random.default_rng(int(seed) + 1)
        model.record(case["steps"], case["every"])
        gauges = np.sort(rng.choice(model.n, size=32, replace=False))
        steps = np.arange(10, case["steps"] + 1, 10)
        model.set_observations(gauges, steps, c.h0[gauges][None, :] * rng.uniform(0.95, 1.05, (steps.size, 32)))
        return {"kind": kind, "model": model, "friction": c.friction[0] * (1.0 + 0.05 * rng.uniform(-1, 1, model.n))}
    if kind == "porosity":
        dt = _step_length(case["cells"])
        c, _ = _inputs("unfrictioned", "muscl_evr", case["cells"], seed)
        c.opts = dict(c.opts, t_max=case["steps"] * dt)
        model = sw2d.SpModel(c)
        rng = np.random.default_rng(int(seed) + 1)
        gauges = np.sort(rng.choice(model.n, size=32, replace=False))
        times = np.arange(1, max(2, case["steps"] // 10 + 1)) * (10 * dt)
        times = times[times <= case["steps"] * dt]
        model.assim_configure(phi_transform="none", cost_normalize=True)
        model.assim_set_gauges(times, gauges, np.ones(32), c.h0[gauges][None, :] * rng.uniform(0.95, 1.05, (times.size, 32)))
        return {"kind": kind, "model": model, "m": np.clip(c.phi + 0.02 * rng.uniform(-1, 1, model.n), 0.05, 1.0),
                "every": case["every"]}
    if kind == "ensemble":
        models = [_model(_member_flow(i), "muscl_evr", n, int(seed) * 64 + i)[0]
                  for i, n in enumerate(_member_sizes(case))]
        batch = sw2d.Batch(models)
        for m in models:
            m.save_point()
        out = torch.empty((3, sum(m.n for m in models)), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return {"kind": kind, "models": models, "batch": batch, "steps": case["steps"], "out": out}
    x, t = _batch_inputs(case["batch"], seed)
    return {"kind": "mlp", "net": _network(seed, 1.0), "x": x, "t": t}


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "forward":
        model = state["model"]
        if "start" in state:
            model.set_state_device(*(v.data_ptr() for v in state["start"]))
            model.set_time(*state["time"])
        else:
            model.restore_point()
        done = model.step(state["steps"])
        if state["host"]:
            h, q, r = model.state()
            return {"h": h, "q": q, "r": r, "steps": done}
        out = state["out"]
        model.get_state_device(*(v.data_ptr() for v in out))
        return {"h": out[0], "q": out[1], "r": out[2], "steps": done}
    if kind == "adjoint":
        model = state["model"]
        model.set_param("friction", state["friction"])
        J, g = model.adjoint()
        return {"J": J, **g}
    if kind == "porosity":
        model, m = state["model"], state["m"]
        steps, segments = model.assim_record(m, state["every"])
        J = model.assim_replay_cost(m)
        g, _ = model.assim_gradient(m, state["every"])
        return {"J": J, "gradient": g, "steps": steps, "segments": segments}
    if kind == "ensemble":
        for m in state["models"]:
            m.restore_point()
        done = state["batch"].step(state["steps"])
        at = 0
        for m in state["models"]:
            m.get_state_device(*(state["out"][k, at:at + m.n].data_ptr() for k in range(3)))
            at += m.n
        return {"states": state["out"], "steps": done}
    net = state["net"]
    loss, g = net.loss_grad(state["x"], state["t"])
    net.adam_step(1e-3)
    return {"loss": loss, "gradient": g, "params": net.params}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
# per cell and time step, with 1.5 internal edges and 3 balance terms per cell: the state read and
# written (48), cell statics, edge statics and lists, each once; and the operations of the
# reference's expressions (a division or square root counted once)
_STEP = {("sp", "muscl_evr"): (188, 590), ("sp", "godunov"): (140, 375), ("dip", "muscl_evr"): (224, 690),
         ("dip", "godunov"): (176, 470), ("ddp", "godunov"): (850, 900)}


def work(case):
    kind = case["kind"]
    if kind == "forward":
        model = case["flow"] if case["flow"] in ("dip", "ddp") else "sp"
        b, f = _STEP[(model, case["scheme"])]
        n = case["cells"] * case["steps"]
        return {"bytes": b * n, "flops": f * n}
    if kind == "closure":
        b, f = _STEP[("dip", "godunov")]
        n = case["cells"] * case["steps"]
        return {"bytes": b * n, "flops": (f + 2 * (10 * 64 + 64 * 64 + 64 * 2)) * n}
    if kind == "adjoint":  # the forward steps again, then their reverse: about twice the operations
        n = case["cells"] * case["steps"]
        return {"bytes": 3 * 188 * n, "flops": 3 * 590 * n}
    if kind == "porosity":  # dry run, replay, recompute and reverse
        n = case["cells"] * case["steps"]
        return {"bytes": 5 * 188 * n, "flops": 5 * 590 * n}
    if kind == "ensemble":
        n = sum(_member_sizes(case)) * case["steps"]
        return {"bytes": 188 * n, "flops": 590 * n}
    n = case["batch"]
    return {"bytes": n * 12 * 4 + 4994 * 4 * 7, "flops": 3 * 2 * (10 * 64 + 64 * 64 + 64 * 2) * n}


# ------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "forward" and case["flow"] != "ddp":
            c, t0 = _inputs(case["flow"], case["scheme"], case["cells"], seed)
            h, q, r, done = _Step(c, t0).run(case["steps"])
            if case["flow"] == "lake":  # the discharges of water at rest are rounding alone
                q = r = None
            return {"h": h, "q": q, "r": r, "steps": done}
        if kind == "ensemble":
            ends = []
            for i, n in enumerate(_member_sizes(case)):
                c, t0 = _inputs(_member_flow(i), "muscl_evr", n, int(seed) * 64 + i)
                ends.append(_Step(c, t0).run(case["steps"]))
            return {"states": torch.stack([torch.cat([e[k] for e in ends]) for k in range(3)]),
                    "steps": np.array([e[3] for e in ends], dtype=np.int64)}
    if kind == "mlp":
        return _exact_training(*_batch_inputs(case["batch"], seed), sw2d.closure.init_params(int(seed)))
    # the porosity tables of the depth-dependent model, the two gradients (their reference defines
    # the adjoint branch by branch) and the network's corrections inside the step have no short
    # restatement: they are held to the start's own values
    return None


def _exact_training(x, t, params):
    p = torch.from_numpy(params.astype(np.float64)).requires_grad_(True)
    shapes, k, w = [(64, 10), (64,), (64, 64), (64,), (2, 64), (2,)], 0, []
    for s in shapes:
        n = int(np.prod(s))
        w.append(p[k:k + n].reshape(s))
        k += n
    a = torch.from_numpy(x.astype(np.float64))
    a = torch.nn.functional.gelu(a @ w[0].T + w[1], approximate="tanh")
    a = torch.nn.functional.gelu(a @ w[2].T + w[3], approximate="tanh")
    y = a @ w[4].T + w[5]
    loss = ((y - torch.from_numpy(t.astype(np.float64))) ** 2).mean()
    loss.backward()
    g = p.grad
    with torch.no_grad():  # Adam's first step
        q = p - 1e-3 * g / (g.abs() + 1e-8)
    return {"loss": loss.item(), "gradient": g.numpy(), "params": q.numpy()}


class _Step:
    """The explicit finite-volume step on a triangle mesh: Riemann states (first order, or MUSCL
    with the evolved reconstruction), HLLC with the bed source, boundary fluxes, CFL time step,
    balance, friction, head loss and the velocity cap; single or dual integral porosity."""

    def __init__(self, c, t0):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def d(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)

        def ix(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.int64)).to(dev)

        m, o = c.mesh, c.opts
        self.n, self.dip = m.cell_nb, c.is_dip
        self.evr = o["num_scheme"] == "muscl_evr"
        self.blend = o["topo_discretization"] == "blending"
        self.law, self.loss = o["model_friction"], o.get("model_singular_head_loss") == "active"
        self.diss = o.get("model_momentum_dissipation") == "active"
        self.cfl, self.dt_max, self.dt_map = float(o["cfl_max"]), float(o["dt_max"]), float(o["dt_map"])
        self.h_min, self.t_max = float(o["h_min"]), float(o["t_max"])
        self.phi_min, self.v_max, self.fr_max = 1e-16, 100.0, float(o.get("fr_max", 100.0))
        self.t, self.dt = t0, 0.0
        self.h, self.q, self.r = d(c.h0), d(c.q0), d(c.r0)
        self.zb, self.area, self.phi, self.b = d(m.cell_z_b), d(m.cell_area), d(c.phi), d(c.boussinesq)
        self.x, self.y = d(m.cell_x), d(m.cell_y)
        self.L, self.R = ix(m.edge_int_cells[:, 0]), ix(m.edge_int_cells[:, 1])
        self.len, self.nx, self.ny = d(m.edge_int_length), d(m.edge_int_nx), d(m.edge_int_ny)
        self.mx, self.my = d(m.edge_int_mx), d(m.edge_int_my)
        self.bc, self.blen, self.bnx, self.bny = ix(m.edge_bnd_cell), d(m.edge_bnd_length), d(m.edge_bnd_nx), d(m.edge_bnd_ny)
        codes = list(c.bc.codes)
        kind = np.array([codes.index(int(k)) for k in m.edge_bnd_code], dtype=np.int64)
        self.series = [(ix(np.flatnonzero(kind == k)), c.bc.types[k], np.asarray(c.bc.times), np.asarray(c.bc.values)[k])
                       for k in range(len(codes)) if np.any(kind == k)]
        self.gi = d(c.phi_g_int) if self.dip else None
        self.gb = d(c.phi_g_bnd) if self.dip else None

        def turned(a):
            rad = np.asarray(a) * math.atan(1.0) / 45.0
            return d(np.cos(rad)), d(np.sin(rad))

        if self.law != "none":
            self.k1, self.k2 = d(c.friction[0]), d(c.friction[1])
            self.fc, self.fs = turned(c.friction[2])
        if self.loss:
            self.hs, self.l1, self.l2 = d(c.head_loss[0]), d(c.head_loss[1]), d(c.head_loss[2])
            self.lc, self.ls = turned(c.head_loss[3])
        if self.diss:
            self.m1, self.m2 = d(c.mu[0]), d(c.mu[1])
            self.mc, self.ms = turned(c.mu[2])
        # w / (area phi) of both sides; the flux kept by edges between dry cells starts at zero
        wet = lambda k, w: torch.where(self.phi[k] > self.phi_min, w / self.area[k] / self.phi[k], torch.zeros_like(w))  # noqa: E731
        self.cL, self.cR, self.cB = wet(self.L, self.len), wet(self.R, self.len), wet(self.bc, self.blen)
        self.flux = [torch.zeros_like(self.len) for _ in range(5)]
        if self.evr:  # each cell's edges in increasing order, and how many
            E = self.L.numel()
            cell = torch.cat([self.L, self.R])
            edge = torch.arange(E, device=cell.device).repeat(2)
            order = torch.argsort(cell * E + edge)
            cell, edge = cell[order], edge[order]
            count = torch.bincount(cell, minlength=self.n)
            first = torch.cumsum(count, 0) - count
            place = torch.arange(cell.numel(), device=cell.device) - first[cell]
            self.count = count
            self.by_place = [(cell[place == k], edge[place == k]) for k in range(int(count.max()))]

    def at_bc(self, times, values):
        return float(np.interp(self.t, times, values))

    def lam(self, b, x, c, u):
        if self.dip:
            root = torch.sqrt((b * x - 1) * b * x * u * u + c * c / x.clamp_min(SMALL))
            return b * x * u - root, b * x * u + root
        root = torch.sqrt((b - 1) * b * u * u + c * c)
        return b * u - root, b * u + root

    def godunov(self, k, nx, ny, x):
        h, q, r = self.h[k], self.q[k], self.r[k]
        qn, rn = q * nx + r * ny, -q * ny + r * nx
        lm, lp = self.lam(self.b[k], x, torch.sqrt(GRAVITY * h), qn / h.clamp_min(SMALL))
        return h + self.zb[k], qn, rn, lm, lp

    def evolved(self, k, left, x, sx, sy):
        h, b, zb, z = self.h[k], self.b[k], self.zb[k], self.h[k] + self.zb[k]
        ql, rl = self.q[k] * self.nx + self.r[k] * self.ny, self.r[k] * self.nx - self.q[k] * self.ny
        hd = h.clamp_min(SMALL)
        ul, vl = ql / hd, rl / hd
        lm, lp = self.lam(b, x, torch.sqrt(GRAVITY * hd), ul)
        hs = 0.0
        for s in (lm, lp):
            s = s.clamp_min(0.0) if left else s.clamp_max(0.0)
            dx = self.mx - self.x[k] - 0.5 * s * self.dt * self.nx
            dy = self.my - self.y[k] - 0.5 * s * self.dt * self.ny
            hs = hs + (z + dx * sx[k] + dy * sy[k] - zb).clamp_min(0.0)
        hr = 0.5 * hs
        lm, lp = self.lam(b, x, torch.sqrt(GRAVITY * hr), hr * ul / hr.clamp_min(SMALL))
        return hr + zb, hr * ul, hr * vl, lm, lp

    def slopes(self):
        z = self.h + self.zb
        sx, sy, ws = torch.zeros_like(z), torch.zeros_like(z), torch.zeros_like(z)
        dx, dy, dz = self.x[self.R] - self.x[self.L], self.y[self.R] - self.y[self.L], z[self.R] - z[self.L]
        dist = torch.sqrt(dx * dx + dy * dy)
        for k in (self.L, self.R):  # the products of two differences have one sign from both sides
            sx.index_add_(0, k, dz * dx / dist / dist / dist)
            sy.index_add_(0, k, dz * dy / dist / dist / dist)
            ws.index_add_(0, k, 1.0 / dist)
        many = self.count > 1
        sx, sy = torch.where(many, sx / ws, 0.0), torch.where(many, sy / ws, 0.0)
        for cell, edge in self.by_place:  # the limiter, edge after edge
            lo, hi = torch.minimum(z[self.L[edge]], z[self.R[edge]]), torch.maximum(z[self.L[edge]], z[self.R[edge]])
            zc, gx, gy = z[cell], sx[cell], sy[cell]
            rec = zc + (self.mx[edge] - self.x[cell]) * gx + (self.my[edge] - self.y[cell]) * gy
            f = torch.where(rec < lo, (lo - zc) / (rec - zc), 1.0)
            f = torch.where(rec > hi, (hi - zc) / (rec - zc), f)
            sx[cell], sy[cell] = gx * f, gy * f
        return sx, sy

    def force(self, b, g, phi, h, u):
        if self.dip:
            x = phi / g.clamp_min(SMALL)
            return (b * h * x * x * u * u + 0.5 * GRAVITY * h * h) * g
        return phi * (b * h * u * u + 0.5 * GRAVITY * h * h)

    def hllc(self, L, R):
        zL, qL, rL, mL, pL = L
        zR, qR, rR, mR, pR = R
        bL, bR, fL, fR, zbL, zbR = self.b[self.L], self.b[self.R], self.phi[self.L], self.phi[self.R], self.zb[self.L], self.zb[self.R]
        g, hm, zero = self.gi, self.h_min, torch.zeros_like(zL)
        hL, hR = zL - zbL, zR - zbR
        if not self.blend and not self.dip:
            hL, hR = hL.clamp_min(0.0), hR.clamp_min(0.0)
        none = ((hL <= hm) & (hR <= hm)) | ((fL <= self.phi_min) & (fR <= self.phi_min))
        lhs = ~none & ((fR <= self.phi_min) | ((hR <= hm) & (zL <= zbR + hm)))
        rhs = ~none & ((fL <= self.phi_min) | ((hL <= hm) & (zR <= zbL + hm)))
        both = ~none & ~lhs & ~rhs
        uL, uR, vL, vR = qL / hL.clamp_min(SMALL), qR / hR.clamp_min(SMALL), rL / hL.clamp_min(SMALL), rR / hR.clamp_min(SMALL)
        L1, L2 = torch.minimum(mL, mR).clamp_max(0.0), torch.maximum(pL, pR).clamp_min(0.0)
        den = (L2 - L1).clamp_min(SMALL)
        if self.dip:
            f1 = (L2 * fL * qL - L1 * fR * qR + L1 * L2 * g * (zR - zL)) / den
            dL = (torch.minimum(zL, zbR) - zbL).clamp_min(0.0)
            dR = (torch.minimum(zR, zbL) - zbR).clamp_min(0.0)
            s2 = g * (-GRAVITY * dL * 0.5 * ((zL - zbR).clamp_min(0.0) + hL)) + g * (GRAVITY * dR * 0.5 * ((zR - zbL).clamp_min(0.0) + hR))
            sL = -L1 * s2 / den + 0.5 * GRAVITY * hL * hL * (g - fL).clamp_max(0.0)
            sR = L2 * s2 / den + 0.5 * GRAVITY * hR * hR * (fR - g).clamp_min(0.0)
            f2 = (L2 * self.force(bL, g, fL, hL, uL) - L1 * self.force(bR, g, fR, hR, uR) + L1 * L2 * (fR * qR - fL * qL)) / den
            f3 = torch.where(f1 >= 0, f1 * (fL / g.clamp_min(SMALL)) * vL, f1 * (fR / g.clamp_min(SMALL)) * vR)
        else:
            least = torch.minimum(fL, fR)
            f1 = least * (L2 * qL - L1 * qR + L1 * L2 * (zR - zL)) / den
            s2 = (fR * hR * hR - fL * hL * hL) * 0.5 + 0.5 * least * (hL + hR) * (zL - zR)
            if self.blend:
                a = torch.where((zbL - zbR).abs() > SMALL, ((zL - zR) / (zbL - zbR)).clamp(0.0, 1.0), zero)
                f1 = a * (least * (L2 * qL - L1 * qR + L1 * L2 * (hR - hL)) / den) + (1.0 - a) * f1
                s2 = a * torch.where(zbL > zbR, fR * hR * (zbL - zbR), fL * hL * (zbL - zbR)) + (1.0 - a) * s2
            s2 = s2 * GRAVITY / den
            sL, sR = -L1 * s2, L2 * s2
            f2 = (L2 * (self.force(bL, g, fL, hL, uL) + sL) - L1 * (self.force(bR, g, fR, hR, uR) - sR) + L1 * L2 * (fR * qR - fL * qL)) / den
            f3 = torch.where(f1 >= 0, bL * f1 * vL, bR * f1 * vR)
        new = [torch.where(both, f, zero) for f in (f1, f2, f3, sL, sR)]
        new[3] = torch.where(lhs, -fL * 0.5 * GRAVITY * hL * hL, new[3])
        new[4] = torch.where(rhs, fR * 0.5 * GRAVITY * hR * hR, new[4])
        moves = (zL - zbL > hm) | (zR - zbR > hm)  # edges between dry sides keep their flux
        self.flux = [torch.where(moves, a, b) for a, b in zip(new, self.flux)]

    def boundary(self, S):
        z, q, r, lm, lp = S
        k = self.bc
        h, b, f = z - self.zb[k], self.b[k], self.phi[k]
        g = self.gb if self.dip else f
        low = h < self.h_min
        q, r, h = (torch.where(low, 0.0, v) for v in (q, r, h))
        hs = h.clamp_min(SMALL)
        c, u, l1 = torch.sqrt(GRAVITY * hs), q / hs, lp.clamp_min(0.0)
        inner = self.force(b, g, f, h, u)
        f1, f2 = torch.zeros_like(h), torch.zeros_like(h)
        for at, kind, times, values in self.series:
            v = self.at_bc(times, values)
            H, F, G, Q = h[at], f[at], g[at], q[at]
            if kind == "fr":
                cc = ((u[at] - 2 * c[at]) / (-v - 2)).clamp_min(0.0)
                a1 = F * (-v * cc) * (cc * cc / GRAVITY)
            elif kind in ("q", "phiWq"):
                x = torch.full_like(H, v)
                if self.dip:
                    x = x / G.clamp_min(SMALL) if kind == "phiWq" else x * F / G.clamp_min(SMALL)
                    hc = (x * x / GRAVITY) ** (1.0 / 3.0)
                    a1 = torch.where(hc >= H, G * 1.5 * torch.sqrt(GRAVITY * hc) * hc, x * G)
                else:
                    hc = (x / F.clamp_min(SMALL) / GRAVITY) ** (1.0 / 3.0)
                    a1 = torch.where(hc >= H, F * 1.5 * torch.sqrt(GRAVITY * hc) * hc, x)
            else:
                raise NotImplementedError(kind)
            f1[at], f2[at] = a1, inner[at] + (a1 - Q * F) * l1[at]
        f3 = torch.where(f1 > 0, 0.0, f1 * r / hs)
        if self.dip:
            f2 = f2 + (f - g).clamp_min(0.0) * 0.5 * GRAVITY * h * h
        return f1, f2, f3

    def step(self):
        ones = torch.ones_like
        xL, xR, xB = ((self.phi[k] / g.clamp_min(SMALL) if self.dip else None)
                      for k, g in ((self.L, self.gi), (self.R, self.gi), (self.bc, self.gb)))
        if self.evr:
            sx, sy = self.slopes()
            L, R = self.evolved(self.L, True, xL, sx, sy), self.evolved(self.R, False, xR, sx, sy)
        else:
            L, R = self.godunov(self.L, self.nx, self.ny, xL), self.godunov(self.R, self.nx, self.ny, xR)
        B = self.godunov(self.bc, self.bnx, self.bny, xB)
        lam = torch.stack([L[3].abs(), L[4].abs(), R[3].abs(), R[4].abs()]).amax(0) * self.len
        lamb = torch.maximum(B[3].abs(), B[4].abs()) * self.blen
        wL, wR, wB = self.h[self.L] > self.h_min, self.h[self.R] > self.h_min, self.h[self.bc] > self.h_min
        swept = torch.zeros_like(self.h)
        swept.index_add_(0, self.bc, torch.where(wB, lamb, 0.0))
        swept.index_add_(0, self.L, torch.where(wL, lam, 0.0))
        swept.index_add_(0, self.R, torch.where(wL | wR, lam, 0.0))
        dt = min(self.dt_max, float((self.cfl * (self.area / swept.clamp_min(SMALL))).min()))
        self.hllc(L, R)
        b1, b2, b3 = self.boundary(B)
        if self.dt_map > SMALL and int((self.t + dt) / self.dt_map) > int(self.t / self.dt_map):
            dt = int((self.t + dt) / self.dt_map) * self.dt_map - self.t
        dt = min(dt, self.t_max - self.t)
        h, q, r = self.h.clone(), self.q.clone(), self.r.clone()
        f1, f2, f3, sL, sR = self.flux
        for k, c, nx, ny, a, p, w in ((self.bc, self.cB, self.bnx, self.bny, b1, b2, b3),
                                      (self.L, -self.cL, self.nx, self.ny, f1, f2 - sL, f3),
                                      (self.R, self.cR, self.nx, self.ny, f1, f2 + sR, f3)):
            h.index_add_(0, k, c * a * dt)
            q.index_add_(0, k, c * (nx * p - ny * w) * dt)
            r.index_add_(0, k, c * (ny * p + nx * w) * dt)
        if self.diss:  # where the depth rose, the discharge increment is reduced
            dq, dr = q - self.q, r - self.r
            a, b = self.m1 * (self.mc * dq + self.ms * dr), self.m2 * (-self.ms * dq + self.mc * dr)
            rose = h > self.h + SMALL
            q = torch.where(rose, q - (self.mc * a - self.ms * b), q)
            r = torch.where(rose, r - (self.ms * a + self.mc * b), r)
        h, q, r = (torch.where(v.abs() < SMALL, 0.0, v) for v in (h, q, r))
        neg = h < 0
        h, q, r = (torch.where(neg, 0.0, v) for v in (h, q, r))
        deep, hs = h > max(self.h_min, SMALL), h.clamp_min(SMALL)
        if self.law != "none":
            u, v = q / hs, r / hs
            ul, vl, un = u * self.fc + v * self.fs, -u * self.fs + v * self.fc, torch.sqrt(u * u + v * v)
            p = hs ** (-4.0 / 3.0)
            k = [self.k1, self.k2] if self.law == "manning" else [1.0 / self.k1, 1.0 / self.k2]
            ul, vl = (w * torch.exp(-GRAVITY * un * kk * kk * p * dt) for w, kk in zip((ul, vl), k))
            q, r = torch.where(deep, (ul * self.fc - vl * self.fs) * h, 0.0), torch.where(deep, (ul * self.fs + vl * self.fc) * h, 0.0)
        if self.loss:
            qx, qy = q * self.lc + r * self.ls, -q * self.ls + r * self.lc
            a = torch.where(h > self.hs, torch.sqrt(qx * qx + qy * qy) / hs, 0.0)
            qx, qy = (torch.where(deep, w * torch.exp(-a * kk * dt), 0.0) for w, kk in ((qx, self.l1), (qy, self.l2)))
            q, r = qx * self.lc - qy * self.ls, qx * self.ls + qy * self.lc
        qn = torch.sqrt(q * q + r * r)
        fact = torch.maximum(qn / (hs * self.v_max), qn / torch.sqrt(GRAVITY * hs) / hs / self.fr_max)
        cap = torch.where((h > self.h_min) & (fact > 1.0), fact, ones(fact))
        self.h, self.q, self.r, self.dt = h, q / cap, r / cap, dt
        self.t += dt

    def run(self, steps):
        done = 0
        while done < steps and self.t < self.t_max:
            self.step()
            done += 1
        return self.h, self.q, self.r, done
