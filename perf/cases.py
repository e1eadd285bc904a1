"""Performance cases: what a program built on this framework has it do.

Every case goes through the public entry points (`Simulation`, `Ensemble`,
`coarsen.snapshot`, `surrogate.Stepper`, `Surrogate.train_step`) on
synthetic sphere microstructures of the repository's configurations:
particles of median radius 4-5 cells at solid fractions 0.1-0.4, tanh
interfaces of width 4, compositions at the common tangent plus noise,
dt = 0.8 of the explicit limit.  `listed` names the sizes that stand for the
range, `draw` gives more of it, `exact` the same results from plain torch
in 64 bits.
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

import phasefield_coarsening_gb300 as ppf
from phasefield_coarsening_gb300 import coarsen, surrogate

DT = 0.8 / (6.0 * 1e-14)             # 0.8 of dx^2 / (6 DL)
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(ppf.__file__)), "weights")
C_SOLID, C_LIQUID = 0.47603, 0.99903   # common tangent of the two parabolas
EDGES = (48, 64, 96, 128)            # ensemble domains


def listed():
    return [
        # the reference's own run in its own precision: a small cube, fields saved every 100 steps
        dict(name="f64_64", kind="step", nz=64, ny=64, nx=64, prec="f64", bc="periodic", steps=100, c_steps=0,
             tuned=False, vf=0.1),
        # the same precision at production size, against which FP32 runs are validated
        dict(name="f64_256", kind="step", nz=256, ny=256, nx=256, prec="f64", bc="periodic", steps=8, c_steps=0,
             tuned=False, vf=0.3),
        # a box cut to a sample's outline: odd edges, closed walls, the solute alone relaxing after the full steps
        dict(name="f64_75x90x101_noflux", kind="step", nz=75, ny=90, nx=101, prec="f64", bc="noflux", steps=20,
             c_steps=10, tuned=False, vf=0.25),
        # a small FP32 domain, where a step is a few microseconds and its launch counts
        dict(name="f32_64", kind="step", nz=64, ny=64, nx=64, prec="f32", bc="periodic", steps=100, c_steps=0,
             tuned=False, vf=0.1),
        # an FP32 cube whose edges are no multiple of any tile, closed walls
        dict(name="f32_250_noflux", kind="step", nz=250, ny=250, nx=250, prec="f32", bc="noflux", steps=20, c_steps=0,
             tuned=False, vf=0.3),
        # the benchmark's grid, with the launch choices that a long run picks once at its start
        dict(name="f32_256_tuned", kind="step", nz=256, ny=256, nx=256, prec="f32", bc="periodic", steps=50, c_steps=0,
             tuned=True, vf=0.3),
        # the long coarsening run: steps, then the tracked microstructure (mean radius, count, energies)
        dict(name="f32_512_coarsen", kind="coarsen", nz=512, ny=512, nx=512, prec="f32", bc="periodic", steps=10,
             c_steps=0, tuned=True, vf=0.2),
        # the drop-in program's loop: host arrays in, a few steps, convergence sums, host arrays out
        dict(name="host_128_f64", kind="host", nz=128, ny=128, nx=128, prec="f64", bc="periodic", steps=4, c_steps=0,
             tuned=False, vf=0.3),
        # analysis of a stored state: observables and the particle size distribution
        dict(name="analysis_256_f32", kind="analysis", nz=256, ny=256, nx=256, prec="f32", bc="periodic", steps=0,
             c_steps=0, tuned=False, vf=0.3),
        # a parameter study: 64 independent cubes of four sizes advanced together
        dict(name="ensemble_64", kind="ensemble", n=64, prec="f32", bc="periodic", steps=20, tuned=True),
        # the learned stepper in its production form: ten network calls, fifty corrector steps, checks and snapshot
        dict(name="surrogate_256_w32", kind="surrogate", nz=256, ny=256, nx=256, bc="periodic", width=32, calls=10,
             steps=50, vf=0.3),
        # one training step of that network on a crop
        dict(name="train_64x128x128_w32", kind="train", nz=64, ny=128, nx=128, bc="periodic", width=32, vf=0.25),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["coarsen", "host", "analysis", "analysis", "ensemble", "ensemble", "surrogate", "train"])
    bc = rng.choice(["periodic", "periodic", "noflux"])
    vf = round(rng.uniform(0.1, 0.32), 3)
    if kind == "ensemble":
        return dict(kind=kind, n=_log_uniform(rng, 4, 64), prec=rng.choice(["f32", "f32", "f64"]), bc=bc,
                    steps=rng.randint(4, 12), tuned=False)
    if kind in ("surrogate", "train"):
        nx = rng.choice([128, 256]) if kind == "surrogate" else 128
        nz, ny = _log_uniform(rng, 16, 200 if kind == "surrogate" else 64), _log_uniform(rng, 16, 200 if kind == "surrogate" else 128)
        if kind == "train":
            return dict(kind=kind, nz=nz, ny=ny, nx=nx, bc="periodic", width=rng.choice([16, 32]), vf=vf)
        return dict(kind=kind, nz=nz, ny=ny, nx=nx, bc="periodic", width=rng.choice([16, 32]), calls=rng.randint(1, 6),
                    steps=rng.randint(5, 50), vf=vf)
    prec = rng.choice(["f32", "f64"]) if kind != "coarsen" else "f32"
    if kind == "host":
        prec = "f64"
    hi = {"step": 300, "coarsen": 400, "host": 200, "analysis": 300}[kind]
    edges = [_log_uniform(rng, 24, hi) for _ in range(3)]
    if rng.random() < 0.4:           # a cube, or edges that are round
        edges = [max(32, (e + 16) // 32 * 32) for e in edges]
    cells = edges[0] * edges[1] * edges[2]
    most = max(2, min(100, int((8e8 if prec == "f32" else 1.2e8) / cells)))
    steps = 0 if kind == "analysis" else rng.randint(1, most) if kind != "host" else rng.randint(1, min(8, most))
    c_steps = rng.randint(1, max(1, most // 2)) if kind == "step" and rng.random() < 0.25 else 0
    return dict(kind=kind, nz=edges[0], ny=edges[1], nx=edges[2], prec=prec, bc=bc, steps=steps, c_steps=c_steps,
                tuned=False, vf=vf)


# ------------------------------------------------------------- inputs ----

def _shape(case):
    return (case["nz"], case["ny"], case["nx"])


def spheres(shape, seed, vf, median=5.0, sigma=0.3, width=4.0, noise=1e-3):
    """etaS, etaL, c (float64 on the GPU): one sphere of lognormal radius in
    each cell of a jittered lattice, max over spheres, periodic."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dev = torch.device("cuda")
    mean_vol = 4.0 / 3.0 * math.pi * median ** 3 * math.exp(4.5 * sigma ** 2)
    a = (mean_vol / vf) ** (1.0 / 3.0)
    k = [max(1, int(round(n / a))) for n in shape]
    h = [n / m for n, m in zip(shape, k)]
    jit = (torch.rand((3, *k), generator=g, device=dev) - 0.5) * 0.3
    R = (median * torch.exp(sigma * torch.randn(k, generator=g, device=dev))).clamp(1.5, 0.62 * min(h))
    ax = [torch.arange(n, device=dev, dtype=torch.float32) + 0.5 for n in shape]
    own = [(x / s).long().clamp(max=m - 1) for x, s, m in zip(ax, h, k)]
    D = torch.full(shape, math.inf, device=dev)
    flat = R.reshape(-1)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                i = [o + d for o, d in zip(own, (dz, dy, dx))]
                w = [q % m for q, m in zip(i, k)]
                lin = (w[0][:, None, None] * k[1] + w[1][None, :, None]) * k[2] + w[2][None, None, :]
                r2 = None
                for q, v in enumerate((2, 1, 0)):
                    # lattice centre of the (unwrapped) cell plus that cell's jitter, minus the voxel
                    base = ((i[v].float() + 0.5) * h[v] - ax[v]).reshape([-1 if v == u else 1 for u in range(3)])
                    d = jit[v].reshape(-1)[lin].mul_(h[v]).add_(base)
                    r2 = d.square_() if r2 is None else r2.add_(d.square_())
                D = torch.minimum(D, r2.sqrt_().sub_(flat[lin]))
    etaS = D.double().mul_(-2.0 / width).tanh_().add_(1.0).mul_(0.5)
    del D
    etaL = 1.0 - etaS
    s2 = etaS * etaS
    hS = s2 / (s2 + etaL * etaL)
    del s2
    c = hS * C_SOLID + (1.0 - hS) * C_LIQUID
    del hS
    c += (torch.rand(shape, generator=g, device=dev, dtype=torch.float64) - 0.5) * (2.0 * noise)
    return etaS, etaL, c


def _fields(case, seed):
    return spheres(_shape(case), seed, case["vf"], median=4.0 if case["kind"] == "coarsen" else 5.0)


def _domains(case):
    rng = np.random.default_rng(0)
    out = []
    for _ in range(case["n"]):
        e, vf = int(rng.choice(EDGES)), float(rng.uniform(0.1, 0.4))
        out.append(((e, e, e), vf))
    return out


def _dom_seed(seed, d):
    return int(seed) * 1009 + d + 1


def _new_sim(case, state, prec=None):
    sim = ppf.Simulation(state[0].shape, ppf.params_default(dt=DT), case["bc"], prec or case["prec"])
    torch.cuda.synchronize()
    sim.upload_device([t.data_ptr() for t in state])
    return sim


class _Out:
    """Device arrays that receive a state: float64 as the library hands it
    over, and float32 where the context computes in FP32."""

    def __init__(self, shape, f32):
        self.d = torch.empty((3, *shape), dtype=torch.float64, device="cuda")
        self.f = torch.empty((3, *shape), dtype=torch.float32, device="cuda") if f32 else None
        self.done = torch.cuda.Event()
        self.done.record()

    def fetch(self, handles, slices):
        self.done.synchronize()      # the previous conversion has read the arrays
        for h, sl in zip(handles, slices):
            rc = ppf.lib().ppf_download_device(h, *[self.d[(f, *sl)].data_ptr() for f in range(3)])
            if rc:
                raise ppf.PPFError(rc, ppf.lib().ppf_last_error().decode())
        if self.f is None:
            return self.d
        self.f.copy_(self.d)
        self.done.record()
        return self.f


def _stats(st, prec):
    """Reductions as numbers; those whose terms are FP32 numbers as such."""
    t = np.float32 if prec == "f32" else float
    return {"mass": st["mass"], "solid_cells": int(st["solid_cells"]), "nonfinite": int(st["nonfinite"]),
            **{k: t(st[k]) for k in ("solid", "free_energy", "sum_dc2", "sum_detaS2", "sum_detaL2")}}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        doms = _domains(case)
        ens = ppf.Ensemble([s for s, _ in doms], ppf.params_default(dt=DT), case["bc"], case["prec"])
        handles, slices, at = [], [], 0
        for d, (shape, vf) in enumerate(doms):
            st = spheres(shape, _dom_seed(seed, d), vf)
            ctx = ctypes.c_void_p()
            if ppf.lib().ppf_ensemble_domain(ens.handle, d, ctypes.byref(ctx)):
                raise RuntimeError("no domain %d" % d)
            torch.cuda.synchronize()
            if ppf.lib().ppf_upload_device(ctx, *[t.data_ptr() for t in st]):
                raise RuntimeError("upload of domain %d failed" % d)
            cells = shape[0] * shape[1] * shape[2]
            handles.append(ctx)
            slices.append((slice(at, at + cells),))
            at += cells
        if case["tuned"]:
            ens.autotune(trial_steps=3)
        return dict(case=case, ens=ens, handles=handles, slices=slices, out=_Out((at,), case["prec"] == "f32"))
    state = _fields(case, seed)
    if kind == "host":
        pin = [torch.empty(_shape(case), dtype=torch.float64, pin_memory=True) for _ in range(6)]
        for p, t in zip(pin, state):
            p.copy_(t)
        sim = ppf.Simulation(_shape(case), ppf.params_default(dt=DT), case["bc"], case["prec"])
        return dict(case=case, sim=sim, src=pin[:3], dst=pin[3:])
    if kind in ("surrogate", "train"):
        sim = _new_sim(case, state, "f32")
        sim.step(100)                # relaxed interfaces, as along a run
        net = surrogate.load(os.path.join(WEIGHTS, "surrogate_w%d_k50.npz" % case["width"]))
        if kind == "train":
            tgt = ppf.Simulation(_shape(case), ppf.params_default(dt=DT), case["bc"], "f32")
            tgt.copy_from(sim)
            tgt.step(50)
            tgt.sync()
            return dict(case=case, net=net, sim=sim, tgt=tgt)
        st = surrogate.Stepper(net, sim, calls=case["calls"], corrector_steps=case["steps"])
        return dict(case=case, net=net, sim=sim, stepper=st, out=_Out(_shape(case), True))
    sim = _new_sim(case, state)
    if case["tuned"]:
        sim.autotune(trial_steps=3)
    if kind == "analysis":
        return dict(case=case, sim=sim)
    return dict(case=case, sim=sim, out=_Out(_shape(case), case["prec"] == "f32"))


# ---------------------------------------------------------------- run ----

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        return {"state": state["out"].fetch(state["handles"], state["slices"])}
    sim = state["sim"]
    if kind == "train":
        loss = state["net"].train_step(sim, state["tgt"], lr=1e-4, want_loss=True)
        return {"loss": np.float32(loss), "params": state["net"].get_params()}
    if kind == "surrogate":
        state["stepper"].cycle()
        return {"state": state["out"].fetch([sim.handle], [()]), "stats": _stats(sim.reduce(), "f32")}
    if kind == "host":
        sim.upload_from(*[t.data_ptr() for t in state["src"]])
        sim.step(case["steps"])
        st = sim.reduce()
        sim.download_into(*[t.data_ptr() for t in state["dst"]])
        return {"state": state["dst"], "stats": _stats(st, case["prec"])}
    if kind == "analysis":
        st = sim.reduce()
        pt = sim.particles(0.5, volumes=True)
        sizes = np.zeros(case["nz"] * case["ny"] * case["nx"] // 256 + 1024, np.int64)   # every particle, then zeros
        sizes[:len(pt["volumes"])] = pt["volumes"]
        return {"stats": _stats(st, case["prec"]), "particles": {**pt, "volumes": sizes}}
    if kind == "coarsen":
        sim.step(case["steps"])
        snap = coarsen.snapshot(sim, case["steps"], DT)
        for k in ("solid_fraction", "free_energy"):
            snap[k] = np.float32(snap[k])
        return {"state": state["out"].fetch([sim.handle], [()]), "snapshot": snap}
    sim.step(case["steps"])
    if case["c_steps"]:
        sim.step_c_only(case["c_steps"])
    st = sim.reduce()
    return {"state": state["out"].fetch([sim.handle], [()]), "stats": _stats(st, case["prec"])}


# --------------------------------------------------------------- work ----

# per cell and step: pass A about 20, fluxes and Laplacians about 60, update about 20 operations
STEP_FLOPS, C_STEP_FLOPS, OBSERVE_FLOPS = 100, 35, 60


def _net_flops(width, out=3):
    return 2.0 * 27 * (5 * width + 4 * width * width + width * out)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(s[0] * s[1] * s[2] for s, _ in _domains(case))
        w = 4 if case["prec"] == "f32" else 8
        return {"bytes": cells * (case["steps"] * 6 * w + 3 * w + 24), "flops": cells * case["steps"] * STEP_FLOPS}
    cells = case["nz"] * case["ny"] * case["nx"]
    if kind == "train":
        # forward, input gradients and weight gradients; every activation written and read twice
        net = _net_flops(case["width"])
        act = 2.0 * (16 + 5 * case["width"])
        return {"bytes": cells * (24 + 4 * act), "flops": cells * 3 * net}
    if kind == "surrogate":
        act = 2.0 * (16 + 5 * case["width"])
        return {"bytes": cells * (case["calls"] * (24 + 2 * act) + case["steps"] * 24 + 5 * 12 + 36),
                "flops": cells * (case["calls"] * _net_flops(case["width"]) + case["steps"] * STEP_FLOPS)}
    w = 4 if case["prec"] == "f32" else 8
    b = case["steps"] * 6 * w + case["c_steps"] * 4 * w + 3 * w   # steps, observables
    f = case["steps"] * STEP_FLOPS + case["c_steps"] * C_STEP_FLOPS + OBSERVE_FLOPS
    if kind in ("step", "coarsen"):
        b += 3 * w + 24              # the state handed over
    if kind == "host":
        b += 48 + 6 * w
    if kind in ("analysis", "coarsen"):
        b += w
    return {"bytes": float(cells * b), "flops": float(cells * f)}


# -------------------------------------------------------------- exact ----

def _nb(u, bc):
    """The six neighbours of every cell (z+, z-, y+, y-, x+, x-)."""
    for d in range(3):
        for s in (-1, 1):
            v = torch.roll(u, s, d)
            if bc == "noflux":
                n = u.shape[d]
                e = n - 1 if s == -1 else 0
                v.select(d, e).copy_(u.select(d, e))
            yield v


def _sums(t):
    return float(t.square().sum())


def _march(eS, eL, c, bc, steps, c_steps):
    """The explicit step in 64 bits; also the sums of the last increments."""
    d = ppf.derive(ppf.params_default(dt=DT))
    p = dict(AS=1e9, AL=1e9, CS=-1e6, CL=1e7, cS0=0.455, cL0=0.978, gamma=1.5)
    t1, t3 = -d.L * d.dt, 0.5 * d.dt * d.h2
    sums = [0.0, 0.0, 0.0]
    for it in range(steps + c_steps):
        s2, l2 = eS * eS, eL * eL
        h = s2 / (s2 + l2)
        A = p["AS"] + (p["AL"] - p["AS"]) * h
        mu = p["AS"] * p["AL"] / A * (c - p["cL0"] + (p["cL0"] - p["cS0"]) * h)
        M = d.ML + (d.MS - d.ML) * h
        dc = torch.zeros_like(c)
        for Mn, mn in zip(_nb(M, bc), _nb(mu, bc)):
            dc += (Mn + M) * (mn - mu)
        dc *= t3
        if it < steps:
            cs = p["cS0"] + mu / p["AS"]
            cl = p["cL0"] + mu / p["AL"]
            drive = 0.5 * p["AS"] * (cs - p["cS0"]) ** 2 + p["CS"] - 0.5 * p["AL"] * (cl - p["cL0"]) ** 2 - p["CL"] - mu * (cs - cl)
            dmu = 2.0 * eS * eL / (s2 + l2) ** 2 * drive
            lapS = sum(_nb(eS, bc)) - 6.0 * eS
            lapL = sum(_nb(eL, bc)) - 6.0 * eL
            dS = t1 * (d.m * eS * (s2 - 1.0 + 2.0 * p["gamma"] * l2) - d.kappa * d.h2 * lapS + eL * dmu)
            dL = t1 * (d.m * eL * (l2 - 1.0 + 2.0 * p["gamma"] * s2) - d.kappa * d.h2 * lapL - eS * dmu)
            eS, eL = eS + dS, eL + dL
            if it == steps - 1:
                sums[1:] = [_sums(dS), _sums(dL)]
        c = c + dc
        if it == steps + c_steps - 1:
            sums[0] = _sums(dc)
    return eS, eL, c, sums


def _observe(eS, eL, c, bc, sums):
    d = ppf.derive(ppf.params_default(dt=DT))
    s2, l2 = eS * eS, eL * eL
    h = s2 / (s2 + l2)
    f0 = s2 * s2 / 4 - s2 / 2 + l2 * l2 / 4 - l2 / 2 + 1.5 * s2 * l2 + 0.25
    gr = sum((n - u) ** 2 for u in (eS, eL) for k, n in enumerate(_nb(u, bc)) if k % 2 == 0)
    mu = 1e9 * (c - 0.978 + 0.523 * h)
    fS, fL = 0.5 * mu * mu / 1e9 - 1e6, 0.5 * mu * mu / 1e9 + 1e7
    F = d.m * f0 + 0.5 * d.kappa * d.h2 * gr + h * fS + (1 - h) * fL
    return {"mass": float(c.sum()), "solid_cells": None, "nonfinite": None, "solid": float(h.sum()),
            "free_energy": float(F.sum()), "sum_dc2": sums[0], "sum_detaS2": sums[1], "sum_detaL2": sums[2]}


def _components(solid, bc):
    """Volumes of the 6-connected components, and the solid/liquid faces."""
    big = solid.numel()
    lab = torch.where(solid, torch.arange(big, device=solid.device).reshape(solid.shape), big)
    while True:
        new = lab
        for n in _nb(lab, bc):
            new = torch.where(solid, torch.minimum(new, n), new)
        ext = torch.cat([new.reshape(-1), new.new_full((1,), big)])
        for _ in range(2):
            new = ext[new]
            ext = torch.cat([new.reshape(-1), new.new_full((1,), big)])
        if torch.equal(new, lab):
            break
        lab = new
    vol = torch.unique(lab[solid], return_counts=True)[1]
    faces = 0
    for k, n in enumerate(_nb(solid.to(torch.int8), bc)):
        if k % 2 == 0:
            faces += int((n.bool() != solid).sum())
    return torch.sort(vol)[0], faces


def _particles(eS32, bc):
    vol, faces = _components(eS32 > 0.5, bc)
    r = float((vol.double() * (3.0 / (4.0 * math.pi))).pow(1.0 / 3.0).sum() / max(1, vol.numel()))
    return {"count": None, "mean_radius": r, "solid_volume": float(vol.sum()),
            "largest_volume": float(vol.max()) if vol.numel() else 0.0, "interface_area": float(faces), "volumes": None}


def _layers(p, width):
    ch, off, out = [16] + [width] * 5 + [16], 0, []
    for ci, co in zip(ch[:-1], ch[1:]):
        W = p[off:off + 27 * ci * co].reshape(27, co, ci)
        off += 27 * ci * co
        out.append((W, p[off:off + co]))
        off += co
    return out


def _network(eS, eL, c, layers, cfg):
    """The network's output (3, z, y, x) in 64 bits, periodic."""
    s2 = eS * eS
    h = s2 / (s2 + eL * eL)
    x = [eS, eL, (c - (cfg["c_liquid"] + (cfg["c_solid"] - cfg["c_liquid"]) * h)) * cfg["in_scale_c"]]
    x += [(e - e.bfloat16().double()) * 256.0 for e in (eS, eL)]
    x = torch.stack(x)
    for i, (W, b) in enumerate(layers):
        co, ci = (3 if i == 5 else W.shape[1]), (5 if i == 0 else W.shape[2])
        y = b[:co, None].expand(co, eS.numel())
        for t in range(27):
            sh = (-(t // 9 - 1), -(t // 3 % 3 - 1), -(t % 3 - 1))
            y = y + W[t, :co, :ci] @ torch.roll(x, sh, (1, 2, 3)).reshape(ci, -1)
        y = y.reshape(co, *eS.shape)
        x = y * torch.sigmoid(y) if i < 5 else y
    return x


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "ensemble":
            parts = []
            for d, (shape, vf) in enumerate(_domains(case)):
                r = _march(*spheres(shape, _dom_seed(seed, d), vf), case["bc"], case["steps"], 0)
                parts.append(torch.stack([u.reshape(-1) for u in r[:3]]))
            return {"state": torch.cat(parts, 1)}
        st = _fields(case, seed)
        if kind == "analysis":
            if case["prec"] == "f32":
                st32 = st[0].float()
            else:
                st32 = st[0]
            return {"stats": _observe(*st, case["bc"], [0.0, 0.0, 0.0]), "particles": _particles(st32, case["bc"])}
        if kind == "coarsen":
            if st[0].numel() * case["steps"] > 2e9:
                return None
            r = _march(*st, case["bc"], case["steps"], 0)
            o, q = _observe(*r[:3], case["bc"], r[3]), _particles(r[0], case["bc"])
            return {"state": torch.stack(r[:3]),
                    "snapshot": {"step": None, "time": case["steps"] * DT, "rbar": q["mean_radius"], "count": None,
                                 "solid_fraction": o["solid"] / st[0].numel(), "mass": o["mass"],
                                 "free_energy": o["free_energy"], "interface_area": q["interface_area"],
                                 "nonfinite": None}}
        if kind in ("step", "host"):
            r = _march(*st, case["bc"], case["steps"], case["c_steps"])
            o = _observe(*r[:3], case["bc"], r[3])
            return {"state": torch.stack(r[:3]) if kind == "step" else list(r[:3]), "stats": o}
        # the network
        if st[0].numel() * case.get("calls", 3) * case["width"] ** 2 > 4e9:
            return None
        z = np.load(os.path.join(WEIGHTS, "surrogate_w%d_k50.npz" % case["width"]), allow_pickle=False)
        cfg = {k: float(z[k]) for k in ("c_solid", "c_liquid", "in_scale_c")}
        scale = torch.tensor(np.asarray(z["out_scale"]) * np.asarray(z["gain"]), device="cuda")[:, None, None, None]
        p = torch.tensor(z["params"], device="cuda").double()
        eS, eL, c, _ = _march(*st, "periodic", 100, 0)
        if kind == "surrogate":
            m0 = c.sum()
            for _ in range(case["calls"]):
                mass = c.sum()
                o = _network(eS, eL, c, _layers(p, case["width"]), cfg) * scale
                eS, eL, c = eS + o[0], eL + o[1], c + o[2]
                c = c + (mass - c.sum()) / c.numel()
            eS, eL, c, sums = _march(eS, eL, c, "periodic", case["steps"], 0)
            c = c + (m0 - c.sum()) / c.numel()
            return {"state": torch.stack([eS, eL, c]), "stats": _observe(eS, eL, c, "periodic", sums)}
    if st[0].numel() > 1.1e6:
        return None
    tgt = _march(eS, eL, c, "periodic", 50, 0)[:3]
    lw = torch.tensor(np.asarray(z["loss_weight"]), device="cuda")[:, None, None, None]
    p = p.requires_grad_(True)
    out = _network(eS, eL, c, _layers(p, case["width"]), cfg)
    want = (torch.stack(tgt) - torch.stack([eS, eL, c])) / scale
    loss = (lw * (out - want) ** 2).sum() / (3.0 * c.numel())
    loss.backward()
    g = p.grad
    new = p.detach() - 1e-4 * g / (g.abs() + 1e-8)
    return {"loss": float(loss.detach()), "params": new}
