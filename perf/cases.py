"""Timed cases of the framework: what its users run, through the public entry
points, from the smallest mesh to the largest of this repository's own
configurations.

Kinds of case
  run      an ``Environment`` started from a given state, stepped ``steps``
           times and read back (pdf, rho, velocity).  ``loop`` steps it one
           ``env.step()`` at a time, as the reference's notebooks do.
  frame    one step of a host-coupled program through the C ABI: page-locked
           pdf in, one step, page-locked pdf, rho and velocity out.
  batch    many independent cases in one ``Batch``: start from given macros,
           run with residual checks, read back.
  train    one forward/backward pass of the warm-start network on a graph of
           ``cells`` cells (loss, output, gradients).
  predict  ``warmstart.predict_cases``: features, potential-flow solve and
           network of several porous cases, from their containers.

Meshes are in lattice units (spacing about 1, dt half the shortest edge), the
units of the reference's notebooks; ``fv`` runs the finite-volume scaled
update with its own stable dt.  A mesh and its containers are built once per
process, as a user's program loads them from a file; the state, the boundary
values, the network's weights and its inputs come from the seed.
"""
import copy
import functools
import math

import numpy as np
import torch

import fvdbm_jax_gb300 as fv
from fvdbm_jax_gb300 import _native as nat
from fvdbm_jax_gb300 import cases as ready
from fvdbm_jax_gb300 import meshgen, warmstart

F32 = np.float32


def _run(name, mesh, cells, steps, scheme="upwind", lattice=9, kernel="auto", fvol=False, loop=False, tau=0.6):
    return {"name": name, "kind": "run", "mesh": mesh, "cells": cells, "steps": steps, "scheme": scheme,
            "lattice": lattice, "kernel": kernel, "fv": fvol, "loop": loop, "tau": tau}


def listed():
    return [
        # the 3,200-triangle lid-driven cavity for its 2,000 steps
        _run("cavity_3k", "cavity", 3_200, 2_000),
        # the same mesh stepped call by call, as the reference's loops do
        _run("cavity_3k_loop", "cavity", 3_200, 200, loop=True),
        # channel with a cylinder at 60k triangles, both flux schemes
        _run("channel_60k", "channel", 60_000, 1_000, tau=0.55),
        _run("channel_60k_lw", "channel", 60_000, 1_000, scheme="lax_wendroff", tau=0.55),
        # the 13-velocity lattice on the same channel
        _run("channel_60k_d2q13", "channel", 60_000, 400, lattice=13, tau=0.7),
        # a porous sample of middling size with the finite-volume update
        _run("porous_250k_fv", "porous", 250_000, 800, fvol=True, tau=0.6),
        # the 1M-triangle porous square: bit-exact default and contracted family
        _run("porous_1m", "porous", 1_000_000, 1_000),
        _run("porous_1m_fast", "porous", 1_000_000, 1_000, kernel="fast"),
        # a host program that exchanges the whole state every step
        {"name": "frame_1m", "kind": "frame", "mesh": "porous", "cells": 1_000_000, "scheme": "upwind", "tau": 0.6},
        # a suite of uneven cavities and porous squares stepped together
        {"name": "batch_24", "kind": "batch", "cases": 24, "low": 2_000, "high": 60_000, "steps": 300, "check": 100,
         "scheme": "upwind"},
        # training pass of the warm-start network
        {"name": "train_500k", "kind": "train", "cells": 500_000},
        # predicted starts of unseen porous samples
        {"name": "predict_6x40k", "kind": "predict", "cases": 6, "cells": 40_000},
    ]


def draw(rng):
    log = lambda a, b: int(math.exp(rng.uniform(math.log(a), math.log(b))))  # noqa: E731
    kind = rng.choice(["run"] * 6 + ["frame", "batch", "train", "predict"])
    if kind == "run":
        mesh = rng.choice(["cavity", "channel", "porous"])
        cells = log(800 if mesh == "cavity" else 3_000, 1_000_000)
        lattice = rng.choice([9, 9, 9, 13])
        fvol = lattice == 9 and rng.random() < 0.25
        kernel = rng.choice(["auto", "auto", "fast"]) if lattice == 9 else "auto"
        steps = max(16, min(2_000, log(50, 2_000), 600_000_000 // cells))
        loop = rng.random() < 0.2
        return {"kind": "run", "mesh": mesh, "cells": cells, "steps": min(steps, 300) if loop else steps,
                "scheme": rng.choice(["upwind", "lax_wendroff"]), "lattice": lattice, "kernel": kernel, "fv": fvol,
                "loop": loop, "tau": round(rng.uniform(0.55, 1.0), 3)}
    if kind == "frame":
        return {"kind": "frame", "mesh": rng.choice(["cavity", "porous"]), "cells": log(3_000, 1_000_000),
                "scheme": rng.choice(["upwind", "lax_wendroff"]), "tau": round(rng.uniform(0.55, 1.0), 3)}
    if kind == "batch":
        return {"kind": "batch", "cases": rng.randint(2, 24), "low": 2_000, "high": log(8_000, 60_000),
                "steps": rng.randint(100, 300), "check": rng.choice([50, 100]),
                "scheme": rng.choice(["upwind", "lax_wendroff"])}
    if kind == "train":
        return {"kind": "train", "cells": log(4_000, 500_000)}
    return {"kind": "predict", "cases": rng.randint(1, 6), "cells": log(5_000, 40_000)}


# ---------------------------------------------------------------------------
# meshes and containers (one build per process)
@functools.lru_cache(maxsize=48)
def _mesher(mesh, cells, seed=0):
    if mesh == "cavity":
        n = int(round(math.sqrt(cells / 2.0))) + 1
        raw, scale = meshgen.cavity(n, seed=seed), ready.cavity_lattice_scale(n)
    elif mesh == "channel":
        raw = meshgen.channel_cylinder(n_target=cells, seed=seed)
        scale = 1.0 / raw.info["h"]
    else:
        porosity = 0.70 if cells >= 400_000 else 0.80
        for k in (400 if cells >= 400_000 else max(4, cells // 3_000), max(3, cells // 8_000), 2):
            try:
                raw = meshgen.porous(n_obstacles=k, n_target=cells, porosity=porosity, seed=seed, gap_cells=1.0)
                break
            except RuntimeError:
                continue
        scale = 1.0 / raw.info["h"]
    raw.points = np.asarray(raw.points, np.float64) * scale
    m = fv.Mesher().import_meshpy(raw)
    m.calc_mesh_properties()
    return m


@functools.lru_cache(maxsize=48)
def _containers(mesh, cells, seed, lattice, scheme, fvol, tau):
    m = _mesher(mesh, cells, seed)
    dt = ready.fv_stable_dt(m, 0.8) if fvol else 0.5 * float(m.face_lengths.min())
    if lattice == 13:
        dt *= 0.5  # its fastest directions move twice as far in a step
    dyn = (fv.D2Q13 if lattice == 13 else fv.D2Q9)(tau, min(dt, tau))
    return (dyn,) + m.to_env(dyn, scheme)


def _boundary(m, mesh, nodes, rng):
    """The case's boundary values on a copy of its nodes."""
    nodes = copy.copy(nodes)
    if mesh == "cavity":
        for mk in (1, 2, 4):
            nodes = m.set_vel_node(nodes, mk, (0.0, 0.0))
        return m.set_vel_node(nodes, 3, (float(rng.uniform(0.05, 0.1)), 0.0))
    for mk in (1, 3, 5):
        nodes = m.set_vel_node(nodes, mk, (0.0, 0.0))
    if mesh == "channel":  # parabolic inlet, open outlet
        nodes = m.set_vel_node(nodes, 4, (0.0, 0.0))
        sel = m.point_markers == 4
        y = m.points[sel, 1] / m.points[:, 1].max()
        v = np.array(nodes.vel)
        v[sel, 0] = 4.0 * float(rng.uniform(0.05, 0.1)) * y * (1.0 - y)
        nodes.vel = v
        return m.set_rho_node(nodes, 2, 1.0)
    nodes = m.set_rho_node(nodes, 4, float(rng.uniform(1.005, 1.02)))
    return m.set_rho_node(nodes, 2, 1.0)


def _macros(m, rng):
    """A smooth random density and velocity field over the cells."""
    c = np.asarray(m.cell_centers, np.float64)
    c = c / max(float(c.max()), 1e-30)
    rho, u, v = (np.zeros(c.shape[0]) for _ in range(3))
    for _ in range(4):
        k = rng.uniform(1.0, 6.0, 2) * 2.0 * np.pi
        p = c @ k + rng.uniform(0.0, 2.0 * np.pi)
        s, t = np.sin(p), np.cos(p)
        rho += 0.002 * s
        u += 0.01 * rng.uniform(-1, 1) * t
        v += 0.01 * rng.uniform(-1, 1) * t
    return (1.0 + rho).astype(F32), np.stack([u, v], 1).astype(F32)


def _state(dyn, m, rng):
    """A pdf near the equilibrium of such a field, as a flow in motion has it."""
    rho, vel = _macros(m, rng)
    eq = np.asarray(dyn.calc_eq(rho[:, None], vel), F32)
    return (eq * (1.0 + 1e-3 * rng.standard_normal(eq.shape, dtype=F32))).astype(F32)


# ---------------------------------------------------------------------------
def _run_inputs(case, seed):
    lattice, fvol = case.get("lattice", 9), case.get("fv", False)
    rng = np.random.default_rng([seed, 1])
    m = _mesher(case["mesh"], case["cells"], 0)
    dyn, c, f, n = _containers(case["mesh"], case["cells"], 0, lattice, case["scheme"], fvol, case["tau"])
    n = _boundary(m, case["mesh"], n, rng)
    return m, dyn, c, f, n, _state(dyn, m, rng)


def _batch_inputs(case, seed):
    """Cavities and porous squares in turn, sizes spread over [low, high]."""
    rng = np.random.default_rng([seed, 2])
    S = case["cases"]
    out, rho, vel = [], [], []
    for s in range(S):
        mesh = "porous" if s % 2 else "cavity"
        cells = int(case["low"] * (case["high"] / case["low"]) ** (s / max(S - 1, 1)))
        m = _mesher(mesh, cells, s)
        dyn, c, f, n = _containers(mesh, cells, s, 9, case["scheme"], False, 0.6 + 0.02 * s)
        out.append((c, f, _boundary(m, mesh, n, rng)))
        r, v = _macros(m, rng)
        rho.append(r)
        vel.append(v)
    return out, np.concatenate(rho), np.concatenate(vel)


@functools.lru_cache(maxsize=4)
def _graph(cells):
    m = _mesher("cavity", cells, 1)
    _, _, f, _ = _containers("cavity", cells, 1, 9, "upwind", False, 0.6)
    n = np.asarray(m.cell_centers).shape[0]
    return n, warmstart.aggregations(f, m.cell_centers, n)


def _train_inputs(case, seed):
    rng = np.random.default_rng([seed, 3])
    n, aggs = _graph(case["cells"])
    x = rng.standard_normal((n, warmstart.NFEAT), dtype=F32)
    t = rng.standard_normal((n, warmstart.NOUT), dtype=F32)
    return x, aggs, t


def _predict_inputs(case, seed):
    rng = np.random.default_rng([seed, 4])
    cs, rin, rout = [], [], []
    for k in range(case["cases"]):
        cells = int(case["cells"] * (0.7 + 0.6 * k / max(case["cases"], 1)))
        m = _mesher("porous", cells, 10 + k)
        dyn, c, f, n = _containers("porous", cells, 10 + k, 9, "upwind", False, 0.8)
        ri, ro = float(rng.uniform(1.01, 1.05)), float(rng.uniform(0.95, 0.99))
        n = copy.copy(n)
        for mk in (1, 3, 5):
            n = m.set_vel_node(n, mk, (0.0, 0.0))
        n = m.set_rho_node(m.set_rho_node(n, 4, ri), 2, ro)
        cs.append((dyn, c, f, n, m))
        rin.append(ri)
        rout.append(ro)
    return cs, rin, rout


def _scaling(cells):
    """Standardisation of the network's features for samples of that size."""
    side = math.sqrt(cells * 0.43 / 0.8)
    mu = np.array([side / 2, side / 2, side / 40, 0.43, 1.03, 0.97, 0.5, 1 / side, 0.0], F32)
    sd = np.array([side / 3, side / 3, side / 40, 0.1, 0.01, 0.01, 0.3, 1 / side, 1 / side], F32)
    return mu, sd


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "frame"):
        m, dyn, c, f, n, pdf = _run_inputs(case, seed)
        env = fv.Environment(c, f, n, kernel=case.get("kernel", "auto"), finite_volume=case.get("fv", False))
        env.init()
        st = {"case": case, "env": env, "pdf": pdf}
        if kind == "frame":
            pin = lambda shape: torch.zeros(shape, dtype=torch.float32).pin_memory().numpy()  # noqa: E731
            N = pdf.shape[0]
            st.update(pdf=pin(pdf.shape), out=pin(pdf.shape), rho=pin((N,)), vel=pin((N, 2)))
            st["pdf"][...] = pdf
        return st
    if kind == "batch":
        cs, rho, vel = _batch_inputs(case, seed)
        b = fv.Batch(cs)
        b.init()
        return {"case": case, "batch": b, "rho": rho, "vel": vel}
    if kind == "train":
        x, aggs, t = _train_inputs(case, seed)
        net = warmstart.MPNN(seed=seed)
        return {"case": case, "net": net, "g": net._upload([warmstart.Sample(x, aggs, t)], True)}
    cs, rin, rout = _predict_inputs(case, seed)
    net = warmstart.MPNN(seed=seed)
    net.x_mu, net.x_sd = _scaling(case["cells"])
    return {"case": case, "net": net, "cases": cs, "rho_in": rin, "rho_out": rout}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        env = state["env"]
        env.cells.pdf = state["pdf"]
        if case["loop"]:
            for _ in range(case["steps"]):
                env = env.step()
        else:
            env.step(case["steps"])
        return {"pdf": env.cells.pdf, "rho": env.cells.rho, "vel": env.cells.vel}
    if kind == "frame":
        L, h = nat.lib(), state["env"].handle
        nat.check(L.fvdbm_set_state(h, nat.fptr(state["pdf"]), None, None, None), h)
        nat.check(L.fvdbm_step(h, 1), h)
        nat.check(L.fvdbm_get_cells(h, nat.fptr(state["out"]), nat.fptr(state["rho"]), nat.fptr(state["vel"]), None), h)
        return {"pdf": state["out"], "rho": state["rho"], "vel": state["vel"]}
    if kind == "batch":
        b = state["batch"]
        b.set_active(np.ones(b.n_cases, np.int32))
        b.set_cells_eq(state["rho"], state["vel"])
        steps, res, status = b.run_to_steady(1e-9, case["check"], case["steps"])
        st = b.state()
        return {"steps": steps, "res": res, "status": status, "pdf": st["pdf"], "rho": st["rho"], "vel": st["vel"]}
    net = state["net"]
    if kind == "train":
        loss = net.loss_and_grads(state["g"])
        return {"loss": loss, "y": state["g"]["y"], "grads": net.G}
    preds, iterations, residual = warmstart.predict_cases(net, state["cases"], state["rho_in"], state["rho_out"])
    return {"predictions": preds, "iterations": iterations, "residual": residual}


# ---------------------------------------------------------------------------
def _step_bytes(cells, q, scheme):
    """Algorithmic traffic of one step: every pdf read and written, each
    cell's face list, each face's geometry (1.5 faces per triangle)."""
    return cells * (8.0 * q + 12.0 + 30.0 + (12.0 if scheme == "lax_wendroff" else 0.0))


def _step_flops(cells, q):
    """Macros, equilibrium, 1.5 face fluxes and their sums, update."""
    return cells * 19.0 * q


def work(case):
    kind = case["kind"]
    if kind == "run":
        N, s, q = case["cells"], case["steps"], case["lattice"]
        # the state in, out and its macros once, then one pass over the data per step
        return {"bytes": s * _step_bytes(N, q, case["scheme"]) + N * (8.0 * q + 12.0), "flops": s * _step_flops(N, q)}
    if kind == "frame":
        N = case["cells"]
        return {"bytes": _step_bytes(N, 9, case["scheme"]) + N * (72.0 + 12.0), "flops": _step_flops(N, 9)}
    if kind == "batch":
        S, lo, hi = case["cases"], case["low"], case["high"]
        N = sum(lo * (hi / lo) ** (s / max(S - 1, 1)) for s in range(S))
        return {"bytes": case["steps"] * _step_bytes(N, 9, case["scheme"]) + N * 96.0,
                "flops": case["steps"] * _step_flops(N, 9)}
    H, Lr = warmstart.HIDDEN, warmstart.LAYERS
    dense = 2.0 * (warmstart.NFEAT * H + Lr * 2 * H * H + H * warmstart.NOUT)
    if kind == "train":
        # per layer h in and out, and in the backward pass h, dh in and dh out
        n = case["cells"]
        return {"bytes": n * (36.0 + 24.0 + 36.0 + Lr * 5 * 4.0 * H), "flops": 3.0 * n * dense}
    n = case["cases"] * case["cells"]
    return {"bytes": n * (1.5 * 41.0 + 24.0 + 20.0 + 12.0 + Lr * 2 * 4.0 * H), "flops": n * dense}


# ---------------------------------------------------------------------------
# the same quantities in 64 bits, written out plainly
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a))).to(_DEV).to(dtype)


class _Plain:
    """One mesh's step in float64: node values by inverse-distance weights,
    ghost values, face fluxes, relaxation and explicit Euler."""

    def __init__(self, dyn, c, f, n, fvol):
        I = torch.int64
        self.q = int(dyn.NUM_QUIVERS)
        self.K = _t(dyn.KSI)
        self.W = _t({9: [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4,
                     13: [3 / 8] + [1 / 12] * 4 + [1 / 16] * 4 + [1 / 96] * 4}[self.q])
        self.c2 = 1.0 / 3.0 if self.q == 9 else 0.5
        self.it, self.dt = 1.0 / float(dyn.tau), float(dyn.delta_t)
        fc, fd = _t(f.stencil_cells_index, I), _t(f.stencil_dists)
        nrm, L = _t(f.n), _t(np.asarray(f.L).reshape(-1, 1))
        self.v = nrm @ self.K.T
        self.vL = self.v * L
        self.lw = f.flux_scheme == "lax_wendroff"
        if self.lw:
            D = fd.sum(1, keepdim=True)
            self.w = fd[:, :1] / D - self.v * self.dt / (2.0 * D)
        self.s0, self.s1 = fc[:, 0].clamp(min=0), fc[:, 1].clamp(min=0)
        self.ghost = []  # (faces, known cells, distance ratio, end nodes) of either side
        nd = _t(f.nodes_index, I)
        for side in (0, 1):
            g = torch.nonzero(fc[:, side] < 0).reshape(-1)
            self.ghost.append((g, fc[g, 1 - side], (fd[g, side] / fd[g, 1 - side])[:, None], nd[g]))
        self.cf, self.cs = _t(c.face_indices, I), _t(c.face_normals)[:, :, None]
        self.ia = (1.0 / _t(np.asarray(c.areas).reshape(-1, 1))) if fvol else None
        t = np.asarray(n.type).reshape(-1)
        self.sets = []
        for kind in (1, 2):
            p = np.flatnonzero(t == kind)
            idx, d = _t(np.asarray(n.cells_index)[p], I), _t(np.asarray(n.cell_dists)[p])
            w = torch.where(idx >= 0, 1.0 / d, torch.zeros_like(d))
            w = (w / w.sum(1, keepdim=True))[:, :, None]
            self.sets.append((kind, _t(p, I), idx.clamp(min=0), w))
        self.np_, self.nr, self.nv = _t(n.pdf), _t(np.asarray(n.rho).reshape(-1, 1)), _t(n.vel)

    def macros(self, f):
        rho = f.sum(1, keepdim=True)
        return rho, (f @ self.K) / rho

    def eq(self, rho, u):
        a, uu, c2 = u @ self.K.T, (u * u).sum(1, keepdim=True), self.c2
        s = 1.0 + a / c2 + a * a / (2 * c2 * c2) - uu / (2 * c2)
        if self.q == 13:
            s = s + a ** 3 / (2 * c2 ** 3) - 3.0 * a * uu / (2 * c2 * c2)
        return self.W * rho * s

    def step(self, f):
        rho, u = self.macros(f)
        eq = self.eq(rho, u)
        for kind, p, idx, w in self.sets:
            if kind == 1:
                self.nr[p] = (rho[idx] * w).sum(1)
            else:
                self.nv[p] = (u[idx] * w).sum(1)
            self.np_[p] = self.eq(self.nr[p], self.nv[p]) + ((f[idx] - eq[idx]) * w).sum(1)
        sides = [f[self.s0], f[self.s1]]
        for side, (g, known, ratio, nd) in enumerate(self.ghost):
            mean = 0.5 * (self.np_[nd[:, 0]] + self.np_[nd[:, 1]])
            sides[side][g] = mean + (mean - f[known]) * ratio
        l, r = sides
        phi = l + (r - l) * self.w if self.lw else torch.where(self.v >= 0, l, r)
        flux = ((phi * self.vL)[self.cf] * self.cs).sum(1)
        if self.ia is not None:
            flux = flux * self.ia
        return f + self.dt * (self.it * (eq - f) - flux), rho, u


def _exact_steps(dyn, c, f, n, fvol, pdf, steps):
    p = _Plain(dyn, c, f, n, fvol)
    x = _t(pdf)
    rho, u = p.macros(x)
    for _ in range(steps):
        x, rho, u = p.step(x)
    return p, x, rho, u


def _bf16(w):
    return torch.as_tensor(w).to(torch.bfloat16).to(torch.float64)


def _sparse(S):
    ip, col, wt, cols = S
    return torch.sparse_csr_tensor(_t(ip, torch.int64), _t(col, torch.int64), _t(wt), size=(len(ip) - 1, int(cols)))


def _network(net, x, stages):
    """(output, activations) of the network on features x in float64."""
    P = [(_bf16(W).to(_DEV), _t(b)) for W, b in net.get_params(rounded=False)]
    z = [x @ P[0][0].T + P[0][1]]
    h, m = [z[0].clamp(min=0)], []
    for (W, b), agg in zip(P[1:-1], stages):
        a = h[-1]
        for M in agg:
            a = M @ a
        m.append(a)
        z.append(torch.cat([h[-1], a], 1) @ W.T + b)
        h.append(h[-1] + z[-1].clamp(min=0))
    return h[-1] @ P[-1][0].T + P[-1][1], P, z, h, m


def _exact_train(case, seed):
    x, aggs, t = _train_inputs(case, seed)
    net = warmstart.MPNN(seed=seed)
    stages = [[(_sparse(st["M"][:3] + (st["cols"],)), _sparse(st["Mt"][:3] + (st["rows"],))) for st in layer]
              for layer in aggs]
    y, P, z, h, m = _network(net, _t(x), [[s[0] for s in layer] for layer in stages])
    e = y - _t(t)
    loss = (e * e).mean()
    d = 2.0 * e / e.numel()
    grads = [[d.T @ h[-1], d.sum(0)]]
    dh = d @ P[-1][0]
    for k in range(len(stages), 0, -1):
        dz = dh * (z[k] > 0)
        grads.insert(0, [dz.T @ torch.cat([h[k - 1], m[k - 1]], 1), dz.sum(0)])
        dx = dz @ P[k][0]
        H = h[0].shape[1]
        back = dx[:, H:]
        for _, Mt in reversed(stages[k - 1]):
            back = Mt @ back
        dh = dh + dx[:, :H] + back
    dz = dh * (z[0] > 0)
    grads.insert(0, [dz.T @ _t(x), dz.sum(0)])
    return {"loss": loss, "y": y, "grads": torch.cat([g.reshape(-1) for pair in grads for g in pair])}


def _potential(c, f, n, m, ri, ro):
    """phi and -grad phi of one case: no flux through walls, phi given on the
    open faces, conjugate gradients in float64 to 1e-13."""
    I = torch.int64
    fc, sd = _t(f.stencil_cells_index, I), _t(f.stencil_dists)
    L, nd = _t(np.asarray(f.L).reshape(-1)), np.asarray(f.nodes_index)
    t, nr = np.asarray(n.type).reshape(-1), np.asarray(n.rho, np.float64).reshape(-1)
    N = np.asarray(m.cell_centers).shape[0]
    inner = (fc[:, 0] >= 0) & (fc[:, 1] >= 0)
    open_ = ~inner & _t((t[nd[:, 0]] == 2) & (t[nd[:, 1]] == 2), torch.bool)
    phib = _t(0.5 * (nr[nd[:, 0]] + nr[nd[:, 1]] - 2.0 * ro) / (ri - ro))
    a, b = fc[inner, 0], fc[inner, 1]
    g = L[inner] / (sd[inner, 0] + sd[inner, 1])
    own = fc.max(1).values
    gb = L[open_] / sd[open_, 0]
    zero = lambda: torch.zeros(N, dtype=torch.float64, device=_DEV)  # noqa: E731
    diag = zero().index_add_(0, a, g).index_add_(0, b, g).index_add_(0, own[open_], gb)
    rhs = zero().index_add_(0, own[open_], gb * phib[open_])
    ar = torch.arange(N, device=_DEV)
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([a, b, ar]), torch.cat([b, a, ar])]), torch.cat([-g, -g, diag]),
                                (N, N)).coalesce().to_sparse_csr()
    phi = zero()
    r = rhs.clone()
    z = r / diag
    p, rz = z.clone(), float(r @ z)
    for _ in range(20_000):
        q = A @ p
        al = rz / float(p @ q)
        phi += al * p
        r -= al * q
        if float(r.norm()) <= 1e-13 * float(rhs.norm()):
            break
        z = r / diag
        new = float(r @ z)
        p = z + (new / rz) * p
        rz = new
    pf = phi[own].clone()
    d0, d1 = sd[inner, 0], sd[inner, 1]
    pf[inner] = (phi[a] * d1 + phi[b] * d0) / (d0 + d1)
    pf[open_] = phib[open_]
    fl = (pf * L)[:, None] * _t(f.n)
    grad = (fl[_t(c.face_indices, I)] * _t(c.face_normals)[:, :, None]).sum(1)
    return phi, -grad / _t(np.asarray(m.cell_areas).reshape(-1, 1)), inner, open_


def _exact_predict(case, seed):
    cs, rin, rout = _predict_inputs(case, seed)
    net = warmstart.MPNN(seed=seed)
    mu, sd = (_t(v) for v in _scaling(case["cells"]))
    out = []
    for (dyn, c, f, n, m), ri, ro in zip(cs, rin, rout):
        phi, grad, inner, open_ = _potential(c, f, n, m, ri, ro)
        cen = _t(m.cell_centers)
        wall = _t(m.face_centers)[~inner & ~open_]
        dist = torch.cat([torch.cdist(x, wall, compute_mode="donot_use_mm_for_euclid_dist").min(1).values
                          for x in cen.split(4096)])
        one = torch.ones_like(phi)
        x = torch.stack([cen[:, 0], cen[:, 1], dist, _t(np.asarray(m.cell_areas).reshape(-1)), ri * one, ro * one, phi,
                         grad[:, 0], grad[:, 1]], 1)
        stages = [[_sparse(st["M"][:3] + (st["cols"],)) for st in layer]
                  for layer in warmstart.aggregations(f, m.cell_centers, cen.shape[0], net.scales)]
        y = _network(net, (x - mu) / sd, stages)[0]
        out.append(y * _t(net.t_sd) + _t(net.t_mu))
    return {"predictions": out, "iterations": None, "residual": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "frame"):
        m, dyn, c, f, n, pdf = _run_inputs(case, seed)
        _, x, rho, u = _exact_steps(dyn, c, f, n, case.get("fv", False), pdf, case.get("steps", 1))
        return {"pdf": x, "rho": rho.reshape(-1) if kind == "frame" else rho, "vel": u}
    if kind == "batch":
        cs, rho, vel = _batch_inputs(case, seed)
        pdfs, rhos, vels, o = [], [], [], 0
        for c, f, n in cs:
            p = _Plain(c.dynamics, c, f, n, False)
            N = np.asarray(c.pdf).shape[0]
            x = p.eq(_t(rho[o:o + N])[:, None], _t(vel[o:o + N]))
            o += N
            for _ in range(case["steps"]):
                x, _, _ = p.step(x)
            r, u = p.macros(x)  # a case that has retired shows the macros of its final pdf
            pdfs.append(x)
            rhos.append(r.reshape(-1))
            vels.append(u)
        return {"steps": None, "res": None, "status": None, "pdf": torch.cat(pdfs), "rho": torch.cat(rhos),
                "vel": torch.cat(vels)}
    if kind == "train":
        return _exact_train(case, seed)
    return _exact_predict(case, seed)
