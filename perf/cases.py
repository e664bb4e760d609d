"""Performance cases: the time step, its options and its adjoint as a user runs them.

A case is one call pattern of the public API over one workload:

* ``step``     a device-resident run: load a checkpoint, ``Session.step(k)``, read the
               particles back.  k is the output interval of a run (1 when every step is
               looked at, 20 for a run that writes now and then).
* ``host``     a host program that owns the particles and the neighbour list (what the
               drop-in's ``simulation_step`` does): upload, one step that takes the
               caller's list, download, list lengths.
* ``adjoint``  a differentiable rollout: forward and backward through
               ``mps_b200.adjoint.Rollout`` with its checkpoints, all gradients returned.

Workloads come from ``mps_b200.workloads``: the 2-D and 3-D dam breaks at l0 from 0.02 m
(a few thousand particles) to 0.0035 m (2.85 million), the shipped example deck, the
driven sloshing tank, surface tension with wetting.  dt follows l0 (dt = 0.1 l0 / (1 m/s),
as the named workloads have it), positions carry a seeded jitter of 1 % of l0 and, in the
2-D runs, seeded velocities.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mps_b200 import _lib
from mps_b200 import workloads as W
from mps_b200.adjoint import Rollout
from mps_b200.session import Session
from mps_b200.types import DUMMY, FLUID, GHOST, WALL, HostParticles

_FIELDS = ("pos", "vel", "pressure", "n", "type", "on_surface")


def listed():
    return [
        # the smallest call: one 2-D step of the coarse dam break, looked at after every step
        dict(name="step2d_small", path="step", deck="dam2d", l0=0.01, prec="fp64", steps=1),
        # an ordinary 2-D run: 20 steps between outputs at l0 = 0.005
        dict(name="run2d_20", path="step", deck="dam2d", l0=0.005, prec="fp64", steps=20),
        # one small 3-D step (a few thousand particles), as in parameter studies and tests
        dict(name="step3d_small", path="step", deck="small3d", l0=0.02, prec="fp64", steps=1),
        # the shipped example deck: velocity-divergence source, pressure clamp, re = 2.1 l0
        dict(name="deck3d_5", path="step", deck="example3d", l0=0.008, prec="fp64", steps=5),
        # surface tension with wetting on an odd-sized dam break
        dict(name="tension3d", path="step", deck="tension3d", l0=0.0133, prec="fp64", steps=2),
        # a mid-size 3-D run in the mixed form
        dict(name="run3d_mid", path="step", deck="dam3d", l0=0.008, prec="mixed", steps=3),
        # the driven sloshing tank, mixed form
        dict(name="sloshing3d", path="step", deck="slosh3d", l0=0.006, prec="mixed", steps=2),
        # 1.17 million particles in FP64
        dict(name="step3d_c1", path="step", deck="dam3d", l0=0.005, prec="fp64", steps=1),
        # the largest: 2.85 million particles in the mixed form
        dict(name="step3d_c2", path="step", deck="dam3d", l0=0.0035, prec="mixed", steps=1),
        # a host program with its own particles and list
        dict(name="host3d", path="host", deck="dam3d", l0=0.01, prec="fp64", steps=1),
        # gradients of a small 2-D rollout (parameter fitting)
        dict(name="adjoint2d", path="adjoint", deck="dam2d", l0=0.01, prec="fp64", steps=8),
        # gradients of a driven 3-D rollout, mixed form
        dict(name="adjoint3d", path="adjoint", deck="slosh3d", l0=0.0095, prec="mixed", steps=4),
    ]


def _log(rng, lo, hi, digits=5):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), digits)


def draw(rng):
    kind = rng.choice(["2d", "2d", "3d", "3d", "3d", "switch", "slosh", "host", "adjoint"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "2d":
        l0 = _log(rng, 0.0035, 0.012)
        return dict(path="step", deck="dam2d", l0=l0, prec=prec, steps=rng.randint(1, 12))
    if kind == "3d":
        l0 = _log(rng, 0.0055, 0.02)
        return dict(path="step", deck="dam3d", l0=l0, prec=prec, steps=rng.randint(1, 3) if l0 > 0.009 else 1)
    if kind == "switch":
        if rng.random() < 0.5:
            return dict(path="step", deck="example3d", l0=0.008, prec=prec, steps=rng.randint(1, 8))
        return dict(path="step", deck="tension3d", l0=_log(rng, 0.009, 0.018), prec=prec, steps=rng.randint(1, 2))
    if kind == "slosh":
        return dict(path="step", deck="slosh3d", l0=_log(rng, 0.0062, 0.015), prec=prec, steps=rng.randint(1, 3))
    if kind == "host":
        return dict(path="host", deck="dam3d", l0=_log(rng, 0.0095, 0.02), prec=prec, steps=1)
    if rng.random() < 0.5:
        return dict(path="adjoint", deck="dam2d", l0=_log(rng, 0.007, 0.012), prec=prec, steps=rng.randint(2, 8))
    return dict(path="adjoint", deck="slosh3d", l0=_log(rng, 0.0095, 0.016), prec=prec, steps=rng.randint(2, 4))


# ---- workloads -------------------------------------------------------------------


def _workload(case, seed):
    deck, l0 = case["deck"], case["l0"]
    if deck == "dam2d":
        wl = W.dambreak("c3", seed=seed, l0=l0, vel_sigma=0.05)
    elif deck == "small3d":
        wl = W.small_dambreak3d(l0=l0, seed=seed)
    elif deck == "example3d":
        wl = W.example_dambreak3d()
        wl.pos = W.jitter_fluid(wl.pos, wl.types, l0, 0.01, seed)
    elif deck == "slosh3d":
        wl = W.sloshing3d(l0=l0, seed=seed)
    else:
        wl = W.dambreak("c1", seed=seed, l0=l0)
        if deck == "tension3d":
            wl.params.update(surface_tension_enabled="1", wetting_angle_SL="60.0")
    if deck not in ("small3d", "example3d"):
        wl.params["dt"] = repr(0.1 * l0)
    return wl


def _sizes(case):
    wl = _workload(case, 0)
    return wl.n, wl.n_fluid, wl.dim


# ---- the measured calls --------------------------------------------------------------


def prepare(case, seed):
    wl = _workload(case, seed)
    cfg = wl.config()
    prec = _lib.PREC_MIXED if case["prec"] == "mixed" else _lib.PREC_FP64
    if case["path"] == "adjoint":
        axis = wl.drive[2]
        roll = Rollout(cfg, wl.dim, wl.pos, wl.types, case["steps"], every=max(1, case["steps"] // 2),
                       precision=prec, drive_axis=axis)
        rng = np.random.Generator(np.random.PCG64(seed + 7))
        u0 = np.where((wl.types == FLUID)[:, None], rng.normal(0.0, 0.05, size=wl.pos.shape), 0.0)
        f64 = dict(dtype=torch.float64, device="cuda")
        st = dict(path="adjoint", roll=roll, u0=torch.tensor(u0, **f64).requires_grad_(),
                  gscale=torch.tensor(1.0, **f64).requires_grad_(),
                  nu=torch.tensor(cfg.viscosity, **f64).requires_grad_(),
                  target=torch.tensor(wl.pos + rng.normal(0.0, 0.01, size=wl.pos.shape), **f64),
                  amp=None, freq=None)
        if wl.drive[0] != 0.0:
            st["amp"] = torch.tensor(wl.drive[0], **f64).requires_grad_()
            st["freq"] = torch.tensor(wl.drive[1], **f64).requires_grad_()
        return st
    hp = HostParticles(wl.dim, wl.pos, wl.vel, wl.types)
    sess = Session(cfg, wl.dim, hp.n, precision=prec)
    if wl.drive[0] != 0.0:
        sess.set_wall_drive(*wl.drive)
    sess.upload(hp)
    sess.compute_initial_params()
    sess.neighbor_search()
    if case["path"] == "host":
        m = cfg.max_neighbors
        nb, cnt = sess.neighbor_list(m)
        return dict(path="host", sess=sess, hp=hp, out=hp.copy(), nb=nb, cnt=cnt, m=m)
    ckpt = torch.empty(sess.state_bytes(), dtype=torch.uint8, device="cuda")
    sess.state_save(ckpt.data_ptr())
    return dict(path="step", sess=sess, ckpt=ckpt, out=hp, steps=case["steps"])


def run(state):
    if state["path"] == "step":
        sess = state["sess"]
        sess.state_load(state["ckpt"].data_ptr())
        sess.step(state["steps"])
        out = sess.download(state["out"])
        return {f: out[f] for f in _FIELDS}
    if state["path"] == "host":
        sess = state["sess"]
        sess.upload(state["hp"])
        sess.step_with_list(state["nb"], state["cnt"], state["m"])
        out = sess.download(state["out"])
        res = {f: out[f] for f in _FIELDS}
        res["count"] = sess.neighbor_counts(state["m"])
        return res
    leaves = [state["u0"], state["gscale"], state["nu"]]
    if state["amp"] is not None:
        leaves += [state["amp"], state["freq"]]
    x, u = state["roll"](*leaves)
    loss = ((x - state["target"]) ** 2).mean() + 1.0e-4 * (u ** 2).mean()
    return [x.detach(), u.detach(), *torch.autograd.grad(loss, leaves)]


def work(case):
    """One pass: the state read and written once, the particles read back; the pair arithmetic of the
    operators, and a single product with the pressure matrix in place of its solve."""
    n, nf, dim = _sizes(case)
    neighbours = 110.0 if dim == 3 else 28.0
    if case["deck"] == "example3d":
        neighbours = 32.0
    state = n * ((4 * dim + 2) * 8.0 + 20.0)
    passes = case["steps"] * (3 if case["path"] == "adjoint" else 1)
    # viscosity, collision, density, source and matrix, product, minimum and gradient
    flops = passes * n * neighbours * (10.0 * dim + 30.0)
    nbytes = 2.0 * state * passes + n * (24.0 * dim + 32.0)
    if case["path"] == "host":
        nbytes += n * (24.0 * dim + 32.0 + 4.0 * neighbours)
    return {"bytes": nbytes, "flops": flops}


# ---- the same step in 64 bits, plain torch --------------------------------------------------

_EXACT_N = 11000


def _pairs(key, live, re):
    """All ordered pairs (i, j), i != j, both live, closer than re."""
    out_i, out_j = [], []
    idx = torch.nonzero(live).flatten()
    k = key[idx]
    for s in range(0, len(idx), 2048):
        d2 = ((k[None, :, :] - k[s:s + 2048, None, :]) ** 2).sum(-1)
        i, j = torch.nonzero(d2 < re * re, as_tuple=True)
        keep = (i + s) != j
        out_i.append(idx[i[keep] + s])
        out_j.append(idx[j[keep]])
    return torch.cat(out_i), torch.cat(out_j)


def _weight(r, re, rmin):
    return torch.where(r < re, re / torch.clamp(r, min=rmin) - 1.0, torch.zeros_like(r))


def _dist(x, i, j):
    return torch.sqrt(((x[j] - x[i]) ** 2).sum(-1))


def _exact_run(cfg, wl, u0, steps, gscale, nu, amp, freq):
    """`steps` time steps on torch tensors; None if a pair collides (an order-dependent update)."""
    dim, l0, dt, rho = wl.dim, cfg.particle_distance, cfg.dt, cfg.density
    re, ren, rmin = cfg.influence_radius_lap, cfg.influence_radius_n, 0.01 * cfg.particle_distance
    f64 = dict(dtype=torch.float64, device="cuda")
    x = torch.tensor(wl.pos, **f64)
    rest = x[:, wl.drive[2]].clone()
    u = u0
    typ = torch.tensor(wl.types, device="cuda")
    fluid, wall, dummy = typ == FLUID, typ == WALL, typ == DUMMY
    fcol = fluid[:, None].to(torch.float64)
    g = torch.tensor([cfg.gravity[d] for d in range(dim)], **f64)
    n = len(typ)
    zero = torch.zeros(n, **f64)
    rl = max(re, ren)
    pi, pj = _pairs(x, typ != GHOST, rl)
    with torch.no_grad():
        d = _dist(x, pi, pj)
        dens = zero.index_add(0, pi, _weight(d, ren, rmin))
        best = int(torch.argmax(torch.where(fluid, dens, -torch.ones_like(dens))))
        n0 = float(dens[best])
        mine = pi == best
        wl_ = _weight(d[mine], re, rmin)
        lam = float((d[mine] ** 2 * wl_).sum() / wl_.sum())
    coeff = 2.0 * dim / (n0 * lam)
    for step in range(steps):
        w = _weight(_dist(x, pi, pj), re, rmin)
        lap = torch.zeros_like(x).index_add(0, pi, (u[pj] - u[pi]) * w[:, None])
        u = u + dt * fcol * (g * gscale + nu * coeff * lap)
        x = x + dt * fcol * u
        if amp is not None:
            t = (step + 1) * dt
            ax = wl.drive[2]
            moving = (wall | dummy)
            om = 2.0 * math.pi * freq
            x = x.clone()
            u = torch.where(moving[:, None], torch.zeros_like(u), u)
            x[:, ax] = torch.where(moving, rest + amp * torch.sin(om * t), x[:, ax])
            u[:, ax] = torch.where(moving, (amp * om * torch.cos(om * t)).expand(n), u[:, ax])
        pi, pj = _pairs(x.detach(), typ != GHOST, rl)
        r = _dist(x, pi, pj)
        if bool(((r < cfg.collision_distance_ratio * l0) & fluid[pi]).any()):
            return None
        dens = zero.index_add(0, pi, _weight(r, ren, rmin))
        surf = fluid & (dens < cfg.surface_threshold * n0)
        unk = (fluid & ~surf) | wall
        row = torch.cumsum(unk.to(torch.int64), 0) - 1
        ne = int(unk.sum())
        w = _weight(r, re, rmin)
        solid = ~dummy[pj]
        diag = zero.index_add(0, pi[solid], coeff * w[solid])
        both = unk[pi] & unk[pj]
        A = torch.zeros(ne * ne, **f64).index_add(0, row[pi[both]] * ne + row[pj[both]], -coeff * w[both])
        A = A.reshape(ne, ne) + torch.diag(diag[unk])
        if cfg.hs_mode == 1:
            dr = x[pj] - x[pi]
            div = zero.index_add(0, pi[solid], (re / r ** 3 * (dr * (u[pj] - u[pi])).sum(-1))[solid])
            b = -(rho / n0 / dt) * div
        else:
            b = cfg.relaxation_coeff * rho / dt ** 2 * (dens - n0) / n0
        b = torch.where(wall, zero, b)
        p = zero.index_put((torch.nonzero(unk).flatten(),), torch.linalg.solve(A, b[unk]))
        del A
        if cfg.clamp_negative_pressure:
            p = torch.where(fluid & (p < 0), zero, p)
        pd = p.detach()
        low = pd.clone().scatter_reduce(0, pi, pd[pj], "amin")
        arg = torch.arange(n, device="cuda")
        hit = pd[pj] == low[pi]
        arg = torch.where(pd == low, arg, arg.scatter(0, pi[hit], pj[hit]))
        pmin = p[arg]
        dr = x[pj] - x[pi]
        r2 = (dr ** 2).sum(-1)
        grad = torch.zeros_like(x).index_add(0, pi, ((p[pj] - pmin[pi]) / r2 * w)[:, None] * dr)
        du = dt * fcol * (-(dim / n0) * grad / rho)
        u = u + du
        x = x + dt * du
        if amp is None:
            u = torch.where((wall | (typ == GHOST))[:, None], torch.zeros_like(u), u)
        lo = torch.tensor([cfg.domain_min[d] - l0 * (cfg.wall_layers + 1) for d in range(dim)], **f64)
        hi = torch.tensor([cfg.domain_max[d] + l0 * (cfg.wall_layers + 1) for d in range(dim)], **f64)
        if bool((fluid[:, None] & ((x < lo) | (x > hi))).any()):
            return None
    return x, u, p, dens


def exact(case, seed):
    if case["deck"] == "tension3d":
        return None
    wl = _workload(case, seed)
    if wl.n > _EXACT_N * (3 if case["deck"] == "example3d" else 1):
        return None
    cfg = wl.config()
    f64 = dict(dtype=torch.float64, device="cuda")
    amp = torch.tensor(wl.drive[0], **f64) if wl.drive[0] != 0.0 else None
    freq = torch.tensor(wl.drive[1], **f64)
    one, nu = torch.tensor(1.0, **f64), torch.tensor(cfg.viscosity, **f64)
    if case["path"] == "adjoint":
        rng = np.random.Generator(np.random.PCG64(seed + 7))
        u0 = torch.tensor(np.where((wl.types == FLUID)[:, None], rng.normal(0.0, 0.05, size=wl.pos.shape), 0.0), **f64)
        target = torch.tensor(wl.pos + rng.normal(0.0, 0.01, size=wl.pos.shape), **f64)
        leaves = [t.requires_grad_() for t in ([u0, one, nu] + ([amp, freq] if amp is not None else []))]
        out = _exact_run(cfg, wl, u0, case["steps"], one, nu, amp, freq)
        if out is None:
            return None
        x, u = out[:2]
        loss = ((x - target) ** 2).mean() + 1.0e-4 * (u ** 2).mean()
        grads = list(torch.autograd.grad(loss, leaves))
        # the velocities of walls and dummies are not a free input: they carry no adjoint
        grads[0] = grads[0] * torch.tensor(wl.types == FLUID, device="cuda")[:, None]
        return [x.detach(), u.detach(), *grads]
    with torch.no_grad():
        out = _exact_run(cfg, wl, torch.tensor(wl.vel, **f64), case["steps"], one, nu, amp, freq)
    if out is None:
        return None
    res = dict(zip(("pos", "vel", "pressure", "n"), out), type=None, on_surface=None)
    if case["path"] == "host":
        res["count"] = None
    return res
