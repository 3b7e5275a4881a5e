"""The workloads this package's speed is measured on.

Each case is what a program using the package has it do between two looks at
the fields: `prepare` builds the engine (or ensemble, or network) from its
seeded initial state and uploads it, `run` advances it by the case's steps
through the public entry points and hands back the device fields. `exact`
restates the same steps in float64 with torch operations only.

Families: explicit Diffusion / Allen-Cahn in 2-D and 3-D ("stencil"),
Cahn-Hilliard with its mass history, Warren1995 dendrites, ADI line solves of
Diffusion and Allen-Cahn, NCGPU with the Ni-Cu database, ensembles of
Warren1995 and Allen-Cahn members, and the surrogate's forward and backward
pass.
"""
from __future__ import annotations

import math
import random
from pathlib import Path

import numpy as np
import torch

from pyphasefield_gb300 import (CahnAllenGB300, CahnHilliardGB300, DiffusionGB300, NCGPUGB300,
                                Warren1995GB300)
from pyphasefield_gb300.ensemble import Ensemble
from pyphasefield_gb300.surrogate import SurrogateNet

TDB = Path(__file__).resolve().parent.parent / "tests" / "golden" / "ncgpu_nicu.tdb"
F64 = torch.float64


def listed():
    return [
        # the smallest grid of the repository's configurations, looked at every
        # 100 steps: launches and host calls count as much as arithmetic
        {"name": "diffusion_256", "family": "stencil", "model": "diffusion", "shape": "256x256",
         "bc": "PERIODIC", "precision": "fp32", "steps": 100},
        # an ordinary grid of odd sides, looked at often
        {"name": "allen_cahn_777x1303", "family": "stencil", "model": "allen_cahn",
         "shape": "777x1303", "bc": "NEUMANN", "precision": "fp32", "steps": 50},
        # a large grid that streams from HBM
        {"name": "diffusion_8192", "family": "stencil", "model": "diffusion",
         "shape": "8192x8192", "bc": "PERIODIC", "precision": "fp32", "steps": 100},
        # a 3-D grid of uneven sides
        {"name": "allen_cahn3d_320x200x250", "family": "stencil", "model": "allen_cahn",
         "shape": "320x200x250", "bc": "NEUMANN", "precision": "fp32", "steps": 100},
        # spinodal decomposition with conserved mass, the mass looked at every 50 steps
        {"name": "cahn_hilliard_256", "family": "cahn_hilliard", "shape": "256x256x256",
         "bc": "PERIODIC", "steps": 50},
        # the benchmark's dendrite
        {"name": "warren_1024", "family": "warren", "shape": "1024x1024", "bc": "NEUMANN",
         "precision": "fp32", "steps": 200},
        # a small dendrite under interactive use: few steps a call
        {"name": "warren_200x300", "family": "warren", "shape": "200x300", "bc": "PERIODIC",
         "precision": "fp32", "steps": 20},
        # Crank-Nicolson ADI in the reference's own precision
        {"name": "diffusion_cn_adi_1024x1400", "family": "adi", "model": "diffusion",
         "shape": "1024x1400", "solver": "crank-nicolson", "precision": "fp64", "steps": 20},
        # semi-implicit ADI Allen-Cahn (a diagonal that varies per cell)
        {"name": "allen_cahn_adi_1500x2000", "family": "adi", "model": "allen_cahn",
         "shape": "1500x2000", "solver": "implicit", "precision": "fp32", "steps": 10},
        # alloy solidification with orientation fields, float64 (the engine's default)
        {"name": "ncgpu_512", "family": "ncgpu", "shape": "512x512", "bc": "PERIODIC",
         "precision": "fp64", "steps": 10},
        # a parameter study: uneven grids stepped together
        {"name": "ensemble_40", "family": "ensemble", "members": 40, "mix": 7, "steps": 100},
        # one gradient evaluation of surrogate training at its defaults
        {"name": "surrogate_train_8x512", "family": "surrogate", "batch": 8, "side": 512},
    ]


# the most cell-steps a drawn case takes, by family (at most a listed case's cost)
_MOST = {"stencil2": 6.0e9, "stencil3": 1.5e9, "cahn_hilliard": 8e8, "warren": 6e8, "adi": 3e7,
         "ncgpu": 5e6}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _shape(rng, nd, lo, hi):
    return [_log_int(rng, lo, hi) for _ in range(nd)]


def _fit(shape, steps, most):
    """Steps cut so that the case stays within `most` cell-steps."""
    return max(1, min(steps, int(most / math.prod(shape))))


def _name(shape):
    return "x".join(str(n) for n in shape)


def draw(rng):
    family = rng.choice(["stencil", "stencil", "stencil", "cahn_hilliard", "warren", "warren",
                         "adi", "adi", "ncgpu", "ensemble", "surrogate"])
    bc = rng.choice(["PERIODIC", "NEUMANN"])
    steps = _log_int(rng, 5, 200)
    if family == "stencil":
        nd = rng.choice([2, 2, 3])
        shape = _shape(rng, 2, 48, 8192) if nd == 2 else _shape(rng, 3, 24, 448)
        prec = rng.choice(["fp32", "fp32", "fp64"])
        most = _MOST["stencil2" if nd == 2 else "stencil3"] / (16 if prec == "fp64" else 1)
        return {"family": family, "model": rng.choice(["diffusion", "allen_cahn"]),
                "shape": _name(shape), "bc": rng.choice([bc, "DIRCHLET"]), "precision": prec,
                "steps": _fit(shape, steps, most)}
    if family == "cahn_hilliard":
        nd = rng.choice([2, 3, 3])
        shape = _shape(rng, nd, 48, 2048) if nd == 2 else _shape(rng, nd, 24, 256)
        return {"family": family, "shape": _name(shape), "bc": bc,
                "steps": _fit(shape, steps, _MOST[family])}
    if family == "warren":
        prec = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        shape = _shape(rng, 2, 64, 4096 if prec == "fp32" else 1024)
        most = _MOST[family] / (24 if prec == "fp64" else 1)
        return {"family": family, "shape": _name(shape), "bc": bc, "precision": prec,
                "steps": _fit(shape, steps, most)}
    if family == "adi":
        shape = _shape(rng, 2, 48, 4096)
        return {"family": family, "model": rng.choice(["diffusion", "allen_cahn"]),
                "shape": _name(shape), "solver": rng.choice(["implicit", "crank-nicolson"]),
                "precision": rng.choice(["fp32", "fp64"]),
                "steps": _fit(shape, _log_int(rng, 2, 20), _MOST[family])}
    if family == "ncgpu":
        shape = _shape(rng, 2, 48, 1024)
        return {"family": family, "shape": _name(shape), "bc": bc,
                "precision": rng.choice(["fp64", "fp64", "fp32"]),
                "steps": _fit(shape, _log_int(rng, 2, 20), _MOST[family])}
    if family == "ensemble":
        return {"family": family, "members": _log_int(rng, 4, 40), "mix": rng.randrange(1 << 16),
                "steps": 2 * _log_int(rng, 5, 50)}
    return {"family": family, "batch": _log_int(rng, 1, 8), "side": 16 * rng.randint(4, 32)}


# ------------------------------------------------------------------ inputs
def _dims(case):
    return [int(n) for n in case["shape"].split("x")]


def _rand(seed, shape, stream=0, normal=False):
    """Seeded float64 numbers on the device, U[0, 1) or N(0, 1)."""
    g = torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + stream)
    f = torch.randn if normal else torch.rand
    return f(tuple(shape), generator=g, device="cuda", dtype=F64)


def _disks(shape, seed, radius, count):
    """Cells inside `count` disks at seeded places: the first about the middle,
    all centred between cells (no cell sits where the gradient vanishes)."""
    r = random.Random(7919 * int(seed) + 1)
    ny, nx = shape
    y = torch.arange(ny, device="cuda", dtype=F64)[:, None]
    x = torch.arange(nx, device="cuda", dtype=F64)[None, :]
    inside = torch.zeros(ny, nx, dtype=torch.bool, device="cuda")
    for k in range(count):
        cy = ny // 2 - 0.5 if k == 0 else r.randrange(8, ny - 8) + 0.5
        cx = nx // 2 - 0.5 if k == 0 else r.randrange(8, nx - 8) + 0.5
        inside |= (y - cy) ** 2 + (x - cx) ** 2 < radius ** 2
    return inside


def _warren_fields(shape, seed):
    """A solid disk of radius 5 (and a second one elsewhere) in undercooled
    liquid of c = 0.40783 +- 1e-3."""
    phi = 1.0 - _disks(shape, seed, 5.0, 2).to(F64)
    return [phi, 0.40783 + 1e-3 * (2 * _rand(seed, shape) - 1)]


def _ncgpu_fields(shape, seed):
    """A solid seed turned by pi / 4 in a melt of Ni-0.408 Cu."""
    inside = _disks(shape, seed, 5.0, 1).to(F64)
    near = _disks(shape, seed, 10.0, 1)
    q1 = torch.where(near, math.cos(math.pi / 8), 1.0).to(F64)
    q4 = torch.where(near, math.sin(math.pi / 8), 0.0).to(F64)
    return [inside, q1, q4, 0.40831 + 1e-3 * (2 * _rand(seed, shape) - 1)]


def _stencil_field(model, shape, seed):
    if model == "diffusion":
        return 0.5 + 0.01 * _rand(seed, shape, normal=True)
    return _rand(seed, shape)


_STENCIL = {"diffusion": (DiffusionGB300, 0.2, {"D": 1.0}, 5.0),
            "allen_cahn": (CahnAllenGB300, 0.1, {}, 1.0)}


def _stencil_dt(case):
    dt = _STENCIL[case["model"]][1]
    # explicit diffusion is stable below 1 / (2 dimensions)
    return 0.15 if case["model"] == "diffusion" and case["shape"].count("x") == 2 else dt


def _engine(cls, fields, **kw):
    """An engine holding `fields`, uploaded and ready to step."""
    sim = cls(dimensions=list(fields[0].shape), **kw)
    sim.initialize_fields_and_imported_data()
    for f, v in zip(sim.fields, fields):
        f.data[(slice(1, -1),) * v.ndim] = v.cpu().numpy()
    sim.simulate(0)
    return sim


def _sides(case):
    r = random.Random(int(case["mix"]))
    return [_log_int(r, 128, 1024) for _ in range(int(case["members"]))]


def _undercooling(case):
    r = random.Random(int(case["mix"]) + 1)
    return [1595.0 - r.uniform(5.0, 40.0) for _ in range(int(case["members"]))]


def _member_fields(m, side, seed):
    if m % 2 == 0:
        return _warren_fields((side, side), 64 * seed + m)
    return [_disks((side, side), 64 * seed + m, 5.0, 2).to(F64)]


def _net_inputs(case, seed):
    """Weights by name, and field pairs one window apart."""
    P, C, E, nb = 16, 192, 384, 9
    K = 2 * P * P
    w, k = {}, [10]

    def add(name, shape, scale):
        k[0] += 1
        w[name] = scale * _rand(seed, shape, k[0], normal=True)

    add("w_in", (C, K), K ** -0.5)
    add("b_in", (C,), 0.02)
    add("w_out", (K, C), 0.1 * C ** -0.5)
    add("b_out", (K,), 0.02)
    for b in range(nb):
        add(f"dw{b}", (C, 9), 1 / 3)
        add(f"bdw{b}", (C,), 0.02)
        add(f"w1_{b}", (E, C), C ** -0.5)
        add(f"b1_{b}", (E,), 0.02)
        add(f"w2_{b}", (C, E), 0.1 * E ** -0.5)
        add(f"b2_{b}", (C,), 0.02)
    n, s = int(case["batch"]), int(case["side"])
    old = torch.stack([torch.stack(_warren_fields((s, s), 64 * seed + b)) for b in range(n)])
    move = _rand(seed, old.shape, 5, normal=True) * torch.tensor([0.05, 0.002], device="cuda",
                                                                  dtype=F64)[:, None, None]
    new = (old + move).clamp(0, 1)
    return w, old.float(), new.float()


_SCALES = (20.0, 500.0)  # 1 / standard deviation of the change of phi and of c


def prepare(case, seed):
    fam, seed = case["family"], int(seed)
    if fam == "stencil" or fam == "adi":
        cls, _, ud, dt = _STENCIL[case["model"]]
        ud = dict(ud, precision=case["precision"])
        kw = dict(dx=1.0, dt=_stencil_dt(case), boundary_conditions=case.get("bc"))
        if fam == "adi":
            ud.update(solver=case["solver"], adi=True)
            kw.update(dt=dt, boundary_conditions="PERIODIC")
        f = _stencil_field(case["model"], _dims(case), seed)
        return {"case": case, "sim": _engine(cls, [f], user_data=ud, **kw)}
    if fam == "cahn_hilliard":
        f = 0.5 + 0.1 * (_rand(seed, _dims(case)) - 0.5)
        return {"case": case, "sim": _engine(CahnHilliardGB300, [f], dx=1.0, dt=0.01,
                                             boundary_conditions=case["bc"],
                                             user_data={"M": 1.0, "epsilon": 1.0})}
    if fam == "warren":
        sim = _engine(Warren1995GB300, _warren_fields(_dims(case), seed), dx=4.6e-8,
                      boundary_conditions=case["bc"],
                      user_data={"seed": seed, "precision": case["precision"]})
    elif fam == "ncgpu":
        sim = _engine(NCGPUGB300, _ncgpu_fields(_dims(case), seed), dx=4.6e-6, tdb_path=str(TDB),
                      temperature_type="ISOTHERMAL", initial_T=1574.0,
                      boundary_conditions=case["bc"],
                      user_data={"seed": seed, "precision": case["precision"]})
    elif fam == "ensemble":
        sims = []
        for m, (s, T) in enumerate(zip(_sides(case), _undercooling(case))):
            f = _member_fields(m, s, seed)
            if m % 2 == 0:
                sims.append(_engine(Warren1995GB300, f, dx=4.6e-8, boundary_conditions="NEUMANN",
                                    user_data={"T": T, "seed": 64 * seed + m}))
            else:
                sims.append(_engine(CahnAllenGB300, f, dx=1.0, dt=0.1,
                                    boundary_conditions="NEUMANN"))
        ens = Ensemble(sims, rows=4, bands=4, persistent=False)
        torch.cuda.synchronize()
        return {"case": case, "ens": ens,
                "start": [[f.clone() for f in s.device_fields()] for s in sims]}
    else:
        w, old, new = _net_inputs(case, seed)
        net = SurrogateNet(delta_scale=_SCALES)
        net.load_params({n: v.cpu().numpy() for n, v in w.items()})
        return {"case": case, "net": net, "old": old, "new": new}
    sim.synchronize()
    return {"case": case, "sim": sim, "start": [f.clone() for f in sim.device_fields()]}


def run(state):
    case = state["case"]
    fam = case["family"]
    if fam == "surrogate":
        net, (b, _, h, w) = state["net"], state["old"].shape
        stream = torch.cuda.current_stream()
        out = net.forward(state["old"], b, h, w, w, stream)
        loss = net.backward(state["old"], state["new"], b, h, w, w, stream)
        return {"out": out, "loss": loss, "grads": net.g}
    if fam == "ensemble":
        ens = state["ens"]
        # every study starts from the seeded states
        with torch.cuda.stream(ens.stream):
            for s, start in zip(ens.sims, state["start"]):
                for f, v in zip(s.device_fields(), start):
                    f.copy_(v)
        ens.step = 0
        ens.simulate(case["steps"])
        return [s.device_fields() for s in ens.sims]
    sim = state["sim"]
    if "start" in state:
        # growth runs start from the seeded state: the front, and with it the
        # work, moves on with every step
        sim.synchronize()
        for f, v in zip(sim.device_fields(), state["start"]):
            f.copy_(v)
        torch.cuda.current_stream().synchronize()
        sim.time_step_counter = 0
    if fam == "cahn_hilliard":
        sim.mass_history.clear()
        sim.simulate(case["steps"])
        return {"fields": sim.device_fields(), "mass": sim.collect_mass_history()}
    sim.simulate(case["steps"])
    return sim.device_fields()


# ------------------------------------------------------------------ work
def work(case):
    """Fields read and written once per pass; floating-point operations of
    every cell and step (the method's own, without halos or random numbers)."""
    fam = case["family"]
    if fam == "surrogate":
        tokens = int(case["batch"]) * (int(case["side"]) // 16) ** 2
        weights = 2 * 512 * 192 + 9 * (2 * 192 * 384 + 9 * 192)
        # forward, and the gradients of inputs and of weights; the first layer
        # has no input gradient
        flops = 2 * tokens * (3 * weights - 512 * 192)
        fields = int(case["batch"]) * 2 * int(case["side"]) ** 2
        return {"bytes": 4 * (2 * fields + 2 * weights) + 4 * tokens * 512, "flops": flops}
    if fam == "ensemble":
        b = f = 0
        for m, s in enumerate(_sides(case)):
            b += s * s * (16 if m % 2 == 0 else 8)
            f += s * s * (150 if m % 2 == 0 else 17)
        return {"bytes": b, "flops": f * case["steps"]}
    shape = _dims(case)
    cells, nd = math.prod(shape), len(shape)
    size = 8 if case.get("precision", "fp32") == "fp64" else 4
    if fam == "stencil":
        ops = 2 * nd + (3 if case["model"] == "diffusion" else 11)
    elif fam == "adi":
        ops = nd * (8 if case["model"] == "diffusion" else 16)
        ops += 4 * nd if case["solver"] == "crank-nicolson" else 0
    else:
        ops = {"cahn_hilliard": 4 * nd + 10, "warren": 150, "ncgpu": 600}[fam]
    fields = {"warren": 2, "ncgpu": 4}.get(fam, 1)
    return {"bytes": 2 * fields * cells * size, "flops": ops * cells * case["steps"]}


# ------------------------------------------------------------------ exact
def _pad(x, bc):
    """One ghost layer per side, axis by axis (corners follow)."""
    for ax in range(x.ndim):
        lo, hi = x.narrow(ax, 0, 1), x.narrow(ax, x.shape[ax] - 1, 1)
        if bc == "PERIODIC":
            lo, hi = hi, lo
        elif bc == "DIRCHLET":
            lo = hi = torch.zeros_like(lo)
        x = torch.cat([lo, x, hi], ax)
    return x


def _inner(x):
    return x[(slice(1, -1),) * x.ndim]


def _lap(x, bc):
    p = _pad(x, bc)
    out = (-2.0 * x.ndim) * x
    for ax in range(x.ndim):
        for k in (0, 2):
            sl = [slice(1, -1)] * x.ndim
            sl[ax] = slice(k, k + x.shape[ax])
            out += p[tuple(sl)]
    return out


def _well(x):
    return 4 * x ** 3 - 6 * x ** 2 + 2 * x


def _exact_stencil(model, x, steps, dt, bc):
    for _ in range(steps):
        if model == "diffusion":
            x = x + dt * _lap(x, bc)
        else:
            x = x + dt * 0.1 * (_lap(x, bc) - 16.0 * _well(x))
    return x


def _exact_cahn_hilliard(x, steps, dt, bc):
    mass = []
    for _ in range(steps):
        x = x + dt * _lap(_well(x) - _lap(x, bc), bc)
        mass.append(x.sum())
    return {"fields": [x - 0.5], "mass": torch.stack(mass)}


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF

    def mul(a, b):
        p, q = a * (b & 0xFFFF), a * (b >> 16)
        return (q + (p >> 16)) >> 16, (p + (q << 16)) & mask

    for _ in range(10):
        hi0, lo0 = mul(c0, 0xD2511F53)
        hi1, lo1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = hi1 ^ c1 ^ k0, lo1, hi0 ^ c3 ^ k1, lo0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _words(shape, per, seed, step, key=0):
    """The generator's words for `per` cells along x sharing one block."""
    ny, nx = shape
    n = -(-nx // per)
    q = torch.arange(n, device="cuda")[None, :].expand(ny, n)
    r = torch.arange(ny, device="cuda")[:, None].expand(ny, n)
    z = torch.zeros_like(q)
    w = _philox(q, r, z + step, z, (seed & 0xFFFFFFFF) ^ key, seed >> 32)
    return [(x >> 8).to(F64) for x in w]


def _uniform(shape, seed, step):
    w = torch.stack(_words(shape, 4, seed, step), -1)
    return w.reshape(shape[0], -1)[:, :shape[1]] * 2.0 ** -24


def _normal(shape, seed, step):
    w = _words(shape, 2, seed, step, 0x5EED0000)
    z = [torch.sqrt(-2 * torch.log((w[2 * k] + 0.5) * 2.0 ** -24))
         * torch.cos(2 * math.pi * (w[2 * k + 1] * 2.0 ** -24)) for k in range(2)]
    return torch.stack(z, -1).reshape(shape[0], -1)[:, :shape[1]]


def _exact_warren(phi, c, steps, bc, seed, T=1574.0):
    """Warren1995 at the engine's default constants."""
    dx, shape = 4.6e-8, phi.shape
    tA, tB, lA, lB, sA, sB = 1728.0, 1358.0, 2350000000.0, 1728000000.0, 0.37, 0.29
    dL, dS, bA, bB, vm, R, ye, alpha = 1e-9, 1e-13, 0.0033, 0.0039, 0.00000742, 8.314, 0.04, 0.3
    dt, d, r2 = dx ** 2 / 5.0 / dL, dx / 0.94, math.sqrt(2)
    e2 = 6 * r2 * sA * d / tA
    wA, wB = 3 * sA / (r2 * tA * d), 3 * sB / (r2 * tB * d)
    mA, mB = tA ** 2 * bA / (6 * r2 * lA * d), tB ** 2 * bB / (6 * r2 * lB * d)

    def g1(f, ax):
        return (f.roll(1, ax) - f.roll(-1, ax)) / (2 * dx)

    def g2(f, ax):
        return (f.roll(1, ax) + f.roll(-1, ax) - 2 * f) / (dx * dx)

    for s in range(steps):
        u = _pad(_uniform(shape, seed, s), "NEUMANN")
        p, q = _pad(phi, bc), _pad(c, bc)
        g = p * p * (1 - p) * (1 - p)
        gp = _well(p)
        HA = wA * gp + 30 * lA * (1 / T - 1 / tA) * g
        HB = wB * gp + 30 * lB * (1 / T - 1 / tB) * g
        pxx, pyy, px, py = g2(p, 0), g2(p, 1), g1(p, 0), g1(p, 1)
        pxy, lap = g1(px, 1), pxx + pyy
        D = dS + p ** 3 * (10 - 15 * p + 6 * p * p) * (dL - dS)
        t = D * vm * q * (1 - q) * (HB - HA) / R
        dc = D * (g2(q, 0) + g2(q, 1)) + g1(D, 0) * g1(q, 0) + g1(D, 1) * g1(q, 1) + t * lap \
            + g1(t, 0) * px + g1(t, 1) * py
        th = torch.atan2(py, px)
        eta, etap = 1 + ye * torch.cos(4 * th), -4 * ye * torch.sin(4 * th)
        etapp, c2, s2 = -16 * (eta - 1), torch.cos(2 * th), torch.sin(2 * th)
        M = (1 - q) * mA + q * mB
        H = (1 - q) * HA + q * HB
        dp = M * (e2 * eta * eta * lap - H + e2 * eta * etap * (s2 * (pyy - pxx) + 2 * c2 * pxy)
                  + 0.5 * e2 * (etap * etap + eta * etapp)
                  * (-2 * s2 * pxy + lap + c2 * (pyy - pxx)))
        dp = dp + M * alpha * (2 * u - 1) * (16 * g) * H
        phi, c = phi + dt * _inner(dp), c + dt * _inner(dc)
    return [phi, c]


def _circulant_solve(b, a, ax):
    """(1 + 2 a) x_i - a (x_{i-1} + x_{i+1}) = b_i, periodic, along an axis."""
    n = b.shape[ax]
    lam = 1 + 2 * a * (1 - torch.cos(2 * math.pi * torch.arange(n // 2 + 1, device="cuda",
                                                                dtype=F64) / n))
    lam = lam.reshape([-1 if k == ax else 1 for k in range(b.ndim)])
    return torch.fft.irfft(torch.fft.rfft(b, dim=ax) / lam, n=n, dim=ax)


def _cyclic_solve(b, diag, a, ax):
    """diag_i x_i - a (x_{i-1} + x_{i+1}) = b_i, periodic, along an axis: the
    rank-one corner correction of Sherman and Morrison on two eliminations."""
    b, d = b.movedim(ax, 0).contiguous(), diag.movedim(ax, 0).clone()
    n = b.shape[0]
    gam = -d[0].clone()
    d[0] -= gam
    d[-1] -= a * a / gam
    rhs = torch.zeros(n, 2, *b.shape[1:], device="cuda", dtype=F64)
    rhs[:, 0] = b
    rhs[0, 1], rhs[-1, 1] = gam, -a
    for i in range(1, n):
        m = a / d[i - 1]
        d[i] -= a * m
        rhs[i] += m * rhs[i - 1]
    rhs[n - 1] /= d[n - 1]
    for i in range(n - 2, -1, -1):
        rhs[i] = (rhs[i] + a * rhs[i + 1]) / d[i]
    x, z = rhs[:, 0], rhs[:, 1]
    k = (x[0] - a / gam * x[-1]) / (1 + z[0] - a / gam * z[-1])
    return (x - k * z).movedim(0, ax)


def _half(x, a, ax):
    return (1 - 2 * a) * x + a * (x.roll(1, ax) + x.roll(-1, ax))


def _exact_adi(case, x):
    cn = case["solver"] == "crank-nicolson"
    for _ in range(case["steps"]):
        if case["model"] == "diffusion":
            a = 0.5 * 5.0 if cn else 5.0
            for ax in (0, 1) if cn else (1, 0):
                x = _circulant_solve(_half(x, a, ax) if cn else x, a, ax)
        else:
            a = 0.05 if cn else 0.1
            for ax in (1, 0):
                x = _half(x, a, ax) if cn else x
                x = _cyclic_solve(x, 1 + 2 * a + 0.8 * (4 * x * x - 6 * x + 2), a, ax)
    return x


def _exact_ncgpu(fields, steps, bc, seed):
    """NCGPU with the Ni-Cu database at T = 1574 (components Cu, Ni)."""
    dx, T = 4.6e-6, 1574.0
    phi, q1, q4, c = fields
    d, idx = 4.0 * dx, 1 / dx
    tm, lat, surf, kin = (1358.0, 1728.0), (1728.0, 2350.0), (0.000029, 0.000037), (0.39, 0.33)
    vm, dL, dS, mq, Hq, ye, beta = 7.42, 1e-5, 1e-9, 40000.0, 1e-7, 0.12, 1.5
    W = [3 * s / (math.sqrt(2) * t * d) for s, t in zip(surf, tm)]
    M = [t * t * b / (6 * math.sqrt(2) * x * d) / 1574.0 for t, b, x in zip(tm, kin, lat)]
    e2 = 6 * math.sqrt(2) * surf[1] * d / tm[1]
    eq2, dt, ln = 0.25 * e2, dx ** 2 / 5.0 / dL / 8, math.log(T)
    cu_s = -13542 + 183.804 * T - 31.38 * T * ln + 3.642e29 * T ** -9
    cu_l = -46.545 + 173.881 * T - 31.38 * T * ln
    ni_s = -5179.159 + 117.854 * T - 22.096 * T * ln - 0.0048407 * T ** 2
    ni_l = 11235.527 + 108.457 * T - 22.096 * T * ln - 0.0048407 * T ** 2 - 0.382318e-20 * T ** 7

    def energy(x, y, cu, ni):
        return x * cu + y * ni + 8.3145 * T * (x * torch.log(x) + y * torch.log(y))

    for s in range(steps):
        y = 1 - c
        gl, gs = energy(c, y, cu_l, ni_l), energy(c, y, cu_s, ni_s)
        dgl = 1e7 * (energy(c + 1e-7, y - 1e-7, cu_l, ni_l) - gl)
        dgs = 1e7 * (energy(c + 1e-7, y - 1e-7, cu_s, ni_s) - gs)
        g = phi * phi * (1 - phi) ** 2
        h = phi ** 3 * (6 * phi * phi - 15 * phi + 10)
        mc = vm * c * (dL + h * (dS - dL)) / (8.314 * T)
        df = (dgl + h * (dgs - dgl)) / vm + (W[0] - W[1]) * g * T \
            + math.sqrt(2 * 8.314 * T / vm) * _normal(phi.shape, seed, s)
        full = {n: _pad(v, bc) for n, v in (("p", phi), ("a", q1), ("b", q4), ("c", c),
                                            ("m", mc), ("f", df))}
        ny, nx = phi.shape

        def at(n, j, i):
            return full[n][1 + j:1 + j + ny, 1 + i:1 + i + nx]

        around = ((0, 1), (0, -1), (1, 0), (-1, 0))

        def div(a, b):
            """div(a grad b), face values averaged."""
            out = 0
            for j, i in around:
                out = out + (a(j, i) + a(0, 0)) * (b(j, i) - b(0, 0))
            return 0.5 * idx * idx * out

        px = 0.5 * idx * (at("p", 0, 1) - at("p", 0, -1))
        py = 0.5 * idx * (at("p", 1, 0) - at("p", -1, 0))
        pxx = (at("p", 0, 1) + at("p", 0, -1) - 2 * phi) * idx * idx
        pyy = (at("p", 1, 0) + at("p", -1, 0) - 2 * phi) * idx * idx
        pxy = 0.25 * idx * idx * (at("p", 1, 1) - at("p", 1, -1) - at("p", -1, 1)
                                  + at("p", -1, -1))
        m2 = torch.clamp(px * px + py * py, min=1e-6)
        m4 = m2 * m2
        ax, ay = (0.5 * idx * (at("a", *u) - at("a", *v)) for u, v in (((0, 1), (0, -1)),
                                                                     ((1, 0), (-1, 0))))
        bx, by = (0.5 * idx * (at("b", *u) - at("b", *v)) for u, v in (((0, 1), (0, -1)),
                                                                     ((1, 0), (-1, 0))))
        turn = {n: idx * torch.sqrt((at("a", *n) - q1) ** 2 + (at("b", *n) - q4) ** 2)
                for n in around}
        mgq = 0.5 * sum(turn.values())
        u, v = q1 * q1 - q4 * q4, 2 * q1 * q4
        sx, sy = u * px - v * py, v * px + u * py
        ux, vx = 2 * q1 * ax - 2 * q4 * bx, 2 * q4 * ax + 2 * q1 * bx
        uy, vy = 2 * q1 * ay - 2 * q4 * by, 2 * q4 * ay + 2 * q1 * by
        sxx, sxy = ux * px + u * pxx - vx * py - v * pxy, uy * px + u * pxy - vy * py - v * pyy
        syx, syy = ux * py + u * pxy + vx * px + v * pxx, uy * py + u * pyy + vy * px + v * pxy
        s4 = sx ** 4 + sy ** 4

        def bend(pn, pnn, pno, po, pon, F, Fn, sxn, syn):
            """One direction of the anisotropy divergence; F = d(s4)/d(p_n) / 2."""
            out = Fn / m2 - F * (2 * pn * pnn + 2 * po * pon) / m4
            out = out - (pnn * s4 + pn * (4 * sx ** 3 * sxn + 4 * sy ** 3 * syn)) / m4
            return out + pn * s4 * (4 * pn ** 3 * pnn + 4 * pn * pnn * po ** 2
                                    + 4 * po * pon * pn ** 2 + 4 * po ** 3 * pon) / (m4 * m4)

        tx = bend(px, pxx, pxy, py, pxy, 2 * sx ** 3 * u + 2 * sy ** 3 * v,
                  6 * sx * sx * sxx * u + 2 * sx ** 3 * ux + 6 * sy * sy * syx * v
                  + 2 * sy ** 3 * vx, sxx, syx)
        ty = bend(py, pyy, pxy, px, pxy, -2 * sx ** 3 * v + 2 * sy ** 3 * u,
                  -6 * sx * sx * sxy * v - 2 * sx ** 3 * vy + 6 * sy * sy * syy * u
                  + 2 * sy ** 3 * uy, sxy, syy)
        dp = e2 * (1 - 3 * ye) * T * (pxx + pyy) + 4 * ye * e2 * T * (tx + ty) \
            - 30 * g * (gs - gl) / vm - _well(phi) * T * (c * W[0] + y * W[1]) \
            - 4 * Hq * T * phi * mgq
        dp = dp * (c * M[0] + y * M[1])
        dc = div(lambda *n: at("m", *n), lambda *n: at("f", *n)) \
            - div(lambda *n: at("m", *n) * at("c", *n), lambda *n: at("f", *n))

        def drift(n, q):
            out = 0
            for at_ in around:
                out = out + 2 * Hq * T * (phi * phi + at("p", *at_) ** 2) \
                    * (at(n, *at_) - q) / torch.clamp(turn[at_], min=beta)
            lap = sum(at(n, *at_) for at_ in around) - 4 * q
            return 0.5 * idx * idx * out + eq2 * idx * idx * lap

        f1, f4 = drift("a", q1), drift("b", q4)
        Mq = mq + (1e-6 - mq) * h
        n1 = q1 + dt * Mq * ((1 - q1 * q1) * f1 - q1 * q4 * f4)
        n4 = q4 + dt * Mq * ((1 - q4 * q4) * f4 - q1 * q4 * f1)
        r = torch.sqrt(n1 * n1 + n4 * n4)
        phi = torch.clamp(phi + dt * dp, 1e-6, 0.999999)
        q1, q4, c = n1 / r, n4 / r, c + dt * dc
    return [phi, q1, q4, c]


def _exact_surrogate(case, seed):
    """The network and its gradients without rounding of the operands."""
    from torch.nn.functional import conv2d, gelu, linear
    w, old, new = _net_inputs(case, seed)
    w = {n: v.float().to(F64).requires_grad_() for n, v in w.items()}
    old, new = old.to(F64), new.to(F64)
    b, _, s, _ = old.shape
    gs, K, C = s // 16, 512, 192

    def patches(f):
        f = f.reshape(b, 2, gs, 16, gs, 16).permute(0, 2, 4, 1, 3, 5)
        return f.reshape(b * gs * gs, K)

    def scaled(f, off, sc):
        o, m = (torch.tensor(t, device="cuda", dtype=F64)[:, None, None] for t in (off, sc))
        return patches((f - o) * m)

    y = linear(scaled(old, (0.5, 0.41), (2.0, 20.0)), w["w_in"], w["b_in"])
    for k in range(9):
        img = y.reshape(b, gs, gs, C).permute(0, 3, 1, 2)
        h = conv2d(img, w[f"dw{k}"].reshape(C, 1, 3, 3), w[f"bdw{k}"], padding=1, groups=C)
        h = h.permute(0, 2, 3, 1).reshape(-1, C)
        h = gelu(linear(h, w[f"w1_{k}"], w[f"b1_{k}"]))
        y = y + linear(h, w[f"w2_{k}"], w[f"b2_{k}"])
    out = linear(y, w["w_out"], w["b_out"])
    diff = out - scaled(new - old, (0.0, 0.0), _SCALES)
    loss = (diff * diff).mean()
    loss.backward()
    return {"out": out.detach(), "loss": loss.detach().reshape(1),
            "grads": {n: v.grad for n, v in w.items()}}


def exact(case, seed):
    fam, seed = case["family"], int(seed)
    if fam == "stencil":
        x = _stencil_field(case["model"], _dims(case), seed)
        return [_exact_stencil(case["model"], x, case["steps"], _stencil_dt(case), case["bc"])]
    if fam == "adi":
        return [_exact_adi(case, _stencil_field(case["model"], _dims(case), seed))]
    if fam == "cahn_hilliard":
        x = 0.5 + 0.1 * (_rand(seed, _dims(case)) - 0.5)
        return _exact_cahn_hilliard(x, case["steps"], 0.01, case["bc"])
    if fam == "warren":
        return _exact_warren(*_warren_fields(_dims(case), seed), case["steps"], case["bc"], seed)
    if fam == "ncgpu":
        return _exact_ncgpu(_ncgpu_fields(_dims(case), seed), case["steps"], case["bc"], seed)
    if fam == "ensemble":
        out = []
        for m, (s, T) in enumerate(zip(_sides(case), _undercooling(case))):
            f = _member_fields(m, s, seed)
            if m % 2 == 0:
                out.append(_exact_warren(*f, case["steps"], "NEUMANN", 64 * seed + m, T))
            else:
                out.append([_exact_stencil("allen_cahn", f[0], case["steps"], 0.1, "NEUMANN")])
        return out
    return _exact_surrogate(case, seed)
