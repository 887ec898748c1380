"""The work that a user of this framework has it do, as cases to be timed.

A simulation is advanced by Simulation.step and its grids are read out at the
dump steps (kind "step"); a host that keeps the particles exchanges them with
the device around each step ("host_loop"); the dump itself weights the
particles to charge, temperature and density grids ("dump"); a start-up
solves for the initial electrostatic field ("poisson"); gradients come from a
forward and a backward pass over a window of steps ("adjoint"); parameter
scans advance many runs together ("ensemble").  Grids, particles per cell,
densities and bunches are those of pdp3_b200.workloads, generated on the GPU.

The FP64 form's results are handed on in FP64.  The cell-local form keeps
particles and their deposits in FP32, so its grids and gradients are handed on
in that type.
"""
import math

import numpy as np
import torch

from pdp3_b200 import api
from pdp3_b200.workloads import (EL_CHARGE, EL_MASS, LIGHT_SPEED, PI, absorbing_layer, courant_dt,
                                 gamma_velocity)

EPSILON0, MAGN_CONST = 8.85e-12, 1.26e-6  # include/constant.h:12, 20
ION_MASS = 1836.0
DEVICE = "cuda"
GRIDS = ("E_r", "E_phi", "E_z", "H_r", "H_phi", "H_z", "J_r", "J_phi", "J_z")
PARTICLE = ("r", "z", "vr", "vphi", "vz")


def _step(name, precision, cells_r, cells_z, ppc, steps, pusher="boris", density=1e17, gamma=0.0,
          sort=0, ramp=0.0, cell=3.90625e-4):
    return {"name": name, "kind": "step", "precision": precision, "cells_r": cells_r,
            "cells_z": cells_z, "ppc": ppc, "steps": steps, "pusher": pusher, "density": density,
            "gamma": gamma, "sort": sort, "ramp": ramp, "cell": cell}


def listed():
    """Twelve cases: the step over its sizes, forms and pushers, and the work around it."""
    return [
        # a first look at a set-up, or a regression test's grid: one step and
        # the whole state read back; launches and waits are all of it
        _step("small_fp64", "fp64", 16, 32, 8, 1, density=1e16, gamma=3.0, cell=1.25e-3),
        # a thermal plasma between two dumps, in both forms: short steps
        _step("thermal_fp64", "fp64", 64, 256, 32, 20, density=1e16, cell=7.8125e-4),
        _step("thermal_fp32", "fp32", 64, 256, 32, 20, density=1e16, cell=7.8125e-4),
        # a bunch driving a wake, the ordinary run, in both forms
        _step("wake_fp64", "fp64", 256, 2048, 64, 5, gamma=5.0),
        _step("wake_fp32", "fp32", 256, 2048, 64, 20, gamma=5.0),
        # the largest run: density ramp, Vay pusher, re-sorted every 20 steps
        _step("large_vay_fp32", "fp32", 512, 4096, 64, 20, "vay", gamma=10.0, sort=20, ramp=0.2,
              cell=1.953125e-4),
        # an odd grid with odd particle counts, Vay, re-sorted
        _step("odd_vay_fp64", "fp64", 101, 299, 21, 10, "vay", density=3e16, gamma=4.0, sort=10),
        # a host program that holds the particles, as the upstream classes do
        {"name": "host_loop_fp64", "kind": "host_loop", "precision": "fp64", "cells_r": 128,
         "cells_z": 1024, "ppc": 16, "steps": 1, "pusher": "boris", "density": 1e17, "gamma": 5.0,
         "sort": 0, "ramp": 0.0, "cell": 3.90625e-4},
        # everything a dump step computes from the particles of the wake run
        {"name": "dump_fp32", "kind": "dump", "precision": "fp32", "cells_r": 256,
         "cells_z": 2048, "ppc": 64, "steps": 0, "pusher": "boris", "density": 1e17, "gamma": 0.0,
         "sort": 0, "ramp": 0.0, "cell": 3.90625e-4},
        # the start-up's electrostatic field on the wake run's grid
        {"name": "poisson", "kind": "poisson", "precision": "fp64", "cells_r": 256,
         "cells_z": 2046, "cell": 3.90625e-4},
        # one gradient: a window of steps forward and its reverse
        {"name": "adjoint", "kind": "adjoint", "precision": "fp32", "cells_r": 64, "cells_z": 512,
         "ppc": 32, "window": 250, "interval": 50, "density": 1e17, "gamma": 5.0,
         "cell": 1.5625e-3},
        # a parameter scan: sixteen runs of different grids and densities
        {"name": "ensemble", "kind": "ensemble", "precision": "fp32", "runs": 16, "scale": 2,
         "steps": 20, "cell": 3.90625e-4},
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the ranges that listed() stands for."""
    kind = rng.choice(["step"] * 6 + ["host_loop", "dump", "poisson", "adjoint", "ensemble"])
    cells_r, cells_z = _between(rng, 12, 400), _between(rng, 24, 3000)
    cell = rng.choice([1.953125e-4, 3.90625e-4, 7.8125e-4])
    if kind == "poisson":
        return {"kind": kind, "precision": "fp64", "cells_r": cells_r,
                "cells_z": rng.choice([126, 254, 510, 1022, 2046]), "cell": cell}
    if kind == "adjoint":
        return {"kind": kind, "precision": "fp32", "cells_r": _between(rng, 24, 64),
                "cells_z": _between(rng, 128, 512), "ppc": rng.randint(4, 32),
                "window": rng.randint(20, 200), "interval": rng.randint(10, 50),
                "density": 10 ** rng.uniform(16, 17), "gamma": rng.uniform(3, 10),
                "cell": 1.5625e-3}
    if kind == "ensemble":
        return {"kind": kind, "precision": "fp32", "runs": rng.randint(2, 16),
                "scale": rng.choice([2, 4, 8]), "steps": rng.randint(4, 20), "cell": cell}
    precision = "fp64" if kind == "host_loop" else rng.choice(["fp64", "fp32", "fp32"])
    most = {"step": 6e7, "host_loop": 4e6, "dump": 6e7}[kind]
    ppc = max(1, min(_between(rng, 2, 64), int(most / (2 * cells_r * cells_z))))
    n = 2 * cells_r * cells_z * ppc
    steps = {"step": max(1, min(20, int(4e8 / n))), "host_loop": 1, "dump": 0}[kind]
    return {"kind": kind, "precision": precision, "cells_r": cells_r, "cells_z": cells_z,
            "ppc": ppc, "steps": steps,
            "pusher": rng.choice(["boris", "boris", "vay", "boris_classic"]),
            "density": 10 ** rng.uniform(15.5, 17),
            "gamma": 0.0 if kind == "dump" else rng.choice([0.0, rng.uniform(3, 10)]),
            "sort": rng.choice([0, 0, 10, 20]) if kind == "step" else 0,
            "ramp": rng.choice([0.0, 0.2]), "cell": cell}


# ------------------------------------------------------------------ inputs


def _geometry(case):
    nr, nz, cell = case["cells_r"] + 1, case["cells_z"] + 1, case["cell"]
    g = {"nr": nr, "nz": nz, "r_size": case["cells_r"] * cell, "z_size": case["cells_z"] * cell}
    g["dr"], g["dz"] = g["r_size"] / (nr - 1), g["z_size"] / (nz - 1)
    g["dt"] = courant_dt(g["dr"], g["dz"])
    layer = max(2, min(10, min(nr, nz) // 6))
    g["pml"] = absorbing_layer(nr, nz, layer)
    return g


def _plasma(case, g, seed):
    """Electrons and protons of a thermal plasma, cell after cell: ppc of each
    in every cell, r with density ~ r, 1 eV electrons, cold protons on the
    electrons' places (the conventions of workloads.thermal_plasma)."""
    nrc, nzc, ppc = g["nr"] - 1, g["nz"] - 1, case["ppc"]
    n, dr, dz = nrc * nzc * ppc, g["dr"], g["dz"]
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    f8 = {"device": DEVICE, "dtype": torch.float64}
    lo = torch.arange(nrc, **f8) * dr
    hi = lo + dr
    lo[0], hi[-1] = dr / 2, g["r_size"] - dr / 2
    za = torch.arange(nzc, **f8) * dz
    zb = za + dz
    za[0], zb[-1] = dz / 2, g["z_size"] - dz / 2
    shape = (nrc, nzc, ppc)
    u = torch.rand(shape, generator=gen, **f8)
    r = torch.sqrt((lo * lo)[:, None, None] + u * (hi * hi - lo * lo)[:, None, None]).reshape(n)
    u = torch.rand(shape, generator=gen, **f8)
    z = (za[None, :, None] + u * (zb - za)[None, :, None]).reshape(n)
    del u
    ramp = case.get("ramp", 0.0) * g["z_size"]
    dens = torch.full_like(za, case["density"])
    if ramp > 0:
        dens = dens * torch.clamp(0.5 * (za + zb) / ramp, max=1.0)
    vol = math.pi * (hi * hi - lo * lo)[:, None] * (zb - za)[None, :]
    w = (vol * dens[None, :] / ppc)[:, :, None].expand(shape).reshape(n).contiguous()
    sig = math.sqrt(EL_CHARGE / EL_MASS)
    v = [torch.randn(n, generator=gen, **f8) * sig for _ in range(3)]
    zero = torch.zeros(n, **f8)
    return [(-1.0, 1.0, r, z, *v, w), (1.0, ION_MASS, r, z, zero, zero, zero, w)]


def _fields(case, g, seed):
    """E and H grids as a run meets them: a few smooth modes of a hundredth of
    the wave-breaking field, and in them the seed."""
    rng = np.random.default_rng(seed)
    nr, nz = g["nr"], g["nz"]
    x, y = np.arange(nr) / (nr - 1), np.arange(nz) / (nz - 1)
    amp = 1e5 * math.sqrt(case.get("density", 1e17) / 1e16)
    out = {}
    for name in ("E_r", "E_phi", "E_z", "H_r", "H_phi", "H_z"):
        a = np.zeros((nr, nz))
        for _ in range(3):
            m, k = rng.integers(1, 6), rng.integers(1, 12)
            rad = np.cos(PI * (m - 0.5) * x) if name.endswith("_z") else np.sin(PI * m * x)
            a += rng.normal() * np.outer(rad, np.sin(PI * k * y))
        out[name] = amp * a / (1.0 if name[0] == "E" else 377.0)
    return out


def _bunch(case, g):
    """An electron bunch injected at z = 0, as the wake run's (64 per cell)."""
    if not case.get("gamma"):
        return None
    radius, length = max(4 * g["dr"], 0.05 * g["r_size"]), max(8 * g["dz"], 0.025 * g["z_size"])
    n = int(round(64 * (radius / g["dr"]) * (length / g["dz"])))
    velocity = gamma_velocity(case["gamma"])
    return {"n": n, "duration": length / velocity, "radius": radius,
            "density": 0.5 * case["density"], "velocity": velocity}


def _simulation(case, seed, fields=True):
    g = _geometry(case)
    sim = api.Simulation(g["r_size"], g["z_size"], g["nr"], g["nz"], g["dt"], pml=g["pml"],
                         pusher=case.get("pusher", "boris"), precision=case["precision"],
                         sort_interval=case.get("sort", 0))
    for s in _plasma(case, g, seed):
        sim.add_species_device(*s)
    b = _bunch(case, g)
    if b:
        sim.add_bunch(-1.0, 1.0, b["n"], b["duration"], b["radius"], b["density"], b["velocity"])
    if fields:
        for name, a in _fields(case, g, seed).items():
            sim.set_field(name, a)
    return sim


def _ensemble_cases(case, seed):
    """The runs of an ensemble: grids, particles per cell, densities and bunch
    energies drawn as workloads.ensemble_params draws them."""
    rng = np.random.default_rng(seed // 1000)
    for r in range(case["runs"]):
        yield {"precision": "fp32",
               "cells_r": (64, 128, 256)[r % 3] // case["scale"],
               "cells_z": (256, 512, 1024)[r // 3 % 3] // case["scale"],
               "ppc": 16 + 3 * r, "density": float(10 ** rng.uniform(15, 17)),
               "gamma": float(rng.uniform(3, 10)), "cell": case["cell"]}, seed + 7 * r


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "poisson":
        g = _geometry(case)
        st["sim"] = api.Simulation(g["r_size"], g["z_size"], g["nr"], g["nz"], g["dt"])
        st["rho"] = _rho(g, seed)
        return st
    if kind == "ensemble":
        st["sims"] = [_simulation(c, s) for c, s in _ensemble_cases(case, seed)]
        st["ensemble"] = api.Ensemble(st["sims"])
        st["ensemble"].set_mode("step_graph")
        torch.cuda.empty_cache()
        return st
    sim = st["sim"] = _simulation(case, seed)
    torch.cuda.empty_cache()  # the library has its own copy of the particles
    st["species"] = list(range(3 if case["gamma"] else 2))
    if kind == "host_loop":
        st["host"] = []
        for s in st["species"]:
            n = sim.species_size(s)
            block = torch.empty((5, n), dtype=torch.float64, pin_memory=True).numpy()
            d = {k: block[j] for j, k in enumerate(PARTICLE)}
            d["alive"] = torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()
            st["host"].append((s, d, d))
    if kind == "adjoint":
        w = max(2, case["cells_r"] // 8)
        z0 = min(case["cells_z"] // 9, case["cells_z"] - w)
        st["adjoint"] = api.Adjoint(sim, case["window"], case["interval"],
                                    (0, w, z0, min(case["cells_z"], z0 + 4 * w)))
    return st


def _rho(g, seed):
    rng = np.random.default_rng(seed)
    x, y = np.arange(g["nr"]) / (g["nr"] - 1), np.arange(g["nz"]) / (g["nz"] - 1)
    rho = sum(rng.normal() * np.outer(np.cos(PI * m * x / 2), np.sin(PI * k * y))
              for m in (1, 3) for k in (1, 2, 5))
    return 1.6e-5 * (rho + 0.1 * rng.normal(size=rho.shape))


# --------------------------------------------------------------------- run


def _typed(case, a):
    t = torch.from_numpy(a)
    return t.to(torch.float32) if case["precision"] == "fp32" else t


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "ensemble":
        state["ensemble"].run(case["steps"])
        return [{k: _typed(case, s.field(k)) for k in ("E_r", "E_z", "J_z")}
                for s in state["sims"]]
    sim = state["sim"]
    if kind == "poisson":
        return {"phi": sim.poisson_solve(state["rho"]), "E_r": sim.field("E_r"),
                "E_z": sim.field("E_z")}
    if kind == "adjoint":
        adj = state["adjoint"]
        loss = adj.forward()
        adj.backward()
        out = {"loss": loss,
               "fields": {k: _typed(case, adj.field(k)) for k in GRIDS[:6]},
               "bunch_velocity": adj.bunch_velocity(2)}
        for s in state["species"]:
            out["species%d" % s] = {k: _typed(case, v) for k, v in adj.species(s).items()}
        return out
    if kind == "dump":
        d = sim.diagnostics()
        # the residual and the neutral plasma's total charge are differences
        # of equal numbers: nothing but rounding is left in them
        return {"rho_electrons": sim.charge_density(1), "rho_ions": sim.charge_density(2),
                "temperature": sim.temperature(0), "density": sim.density(0),
                "density_ions": sim.density(1), "E_z": sim.probe("E_z", "frame", 0, 0,
                                                                 sim.nr, sim.nz),
                "field_energy": d["field_energy"], "kinetic_energy": d["kinetic_energy"],
                "rho_norm": d["gauss_norm"], "alive": d["alive"]}
    sim.step(case["steps"])
    if kind == "host_loop":
        sim.exchange_all(state["host"])
        return {"species": [{k: a for k, a in d.items()} for _, d, _ in state["host"]],
                "E_z": sim.field("E_z")}
    sim.sync()
    out = {k: _typed(case, sim.field(k)) for k in GRIDS}
    if case["cells_r"] * case["cells_z"] * case["ppc"] <= 10000 and not case["sort"]:
        for s in state["species"]:  # a small state is read back whole
            p = sim.species(s)
            out["species%d" % s] = {k: _typed(case, p[k]) for k in PARTICLE}
            out["alive%d" % s] = p["alive"]
    return out


def work(case):
    """Bytes: each particle's state read and written once per step (88 B in the
    FP64 form, 52 B in the cell-local one) and each node's fields; flops: the
    arithmetic of gather, push and deposition, about 400 per particle-step."""
    kind, fp32 = case["kind"], case["precision"] == "fp32"
    if kind == "ensemble":
        parts = [work(dict(c, kind="step", steps=case["steps"]))
                 for c, _ in _ensemble_cases(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nodes = (case["cells_r"] + 1) * (case["cells_z"] + 1)
    if kind == "poisson":
        length = 2 * nodes / (case["cells_r"] + 1)
        return {"bytes": 32.0 * nodes, "flops": 2 * 5 * nodes * math.log2(length)}
    n = 2 * case["cells_r"] * case["cells_z"] * case["ppc"]
    if case["gamma"]:
        n += _bunch(case, _geometry(case))["n"]
    if kind == "dump":
        return {"bytes": n * (28.0 if fp32 else 48.0) + 7 * 8.0 * nodes, "flops": 100.0 * n}
    grid = 8.0 * 22 * nodes  # E, H, J and sigma read, E, H and the half-step H written
    if kind == "adjoint":  # the steps forward, and each particle's adjoints back
        step = 52.0 * n + grid
        back = (29.0 + 20 + 20 + 16) * n + 2 * grid
        return {"bytes": case["window"] * (step + back), "flops": 1600.0 * n * case["window"]}
    b = case["steps"] * (n * (52.0 if fp32 else 88.0) + grid)
    if kind == "host_loop":
        b += 2 * 40.0 * n
    return {"bytes": b, "flops": 400.0 * n * case["steps"]}


# ------------------------------------------------------- the same in 64 bits
# The step in cell units (x = r / dr, y = z / dz) with plain torch in FP64:
# the upstream's discretisation (src/particles.cpp, src/eField.cpp,
# src/hField.cpp, src/geometry.cpp:56-107), every difference of large numbers
# formed from in-cell offsets.


def _sigma(g):
    nr, nz, dr, dz, rs, zs = (g[k] for k in ("nr", "nz", "dr", "dz", "r_size", "z_size"))
    l1, l2, l3, s1, s2 = g["pml"]
    left, right, ext = dz * math.floor(nz * l1), dz * math.floor(nz * l2), dr * math.floor(nr * l3)
    i, k = np.arange(nr)[:, None] * np.ones((1, nz)), np.ones((nr, 1)) * np.arange(nz)[None, :]
    sig = np.zeros((nr, nz))
    sig = np.where(dz * k < left, s1 + (s2 - s1) / left ** 2 * (left - dz * k) ** 2, sig)
    sig = np.where(zs - dz * k < right,
                   s1 + (s2 - s1) / right ** 2 * (dz * (k + 1) - zs + right) ** 2, sig)
    corner = ((rs - dr * i <= ext) & (rs - dr * (i + 1) < ext * dz * k / left) &
              (rs - dr * i <= ext / right * (zs - dz * k)))
    return np.where(corner, s1 + (s2 - s1) / ext ** 2 * (dr * (i + 1) - rs + ext) ** 2, sig)


def _radical_inverse(n, base):
    idx, out, scale = np.arange(n), np.zeros(n), 1.0 / base
    while idx.any():
        out += idx % base * scale
        idx, scale = idx // base, scale / base
    return out


def _bunch_state(b, g):
    """Radii and weights of a bunch (src/bunch.cpp:6-80)."""
    dr, dz = g["dr"], g["dz"]
    r = (b["radius"] - dr) * _radical_inverse(b["n"], 9) + dr / 2
    mean = np.where(r > dr, 2 * PI * r * dr * dz, PI * r * r * dz).sum() / b["n"]
    vol = np.where(r > dr / 2, 2 * PI * r * dr * dz, PI * (r * r + r * dr + dr * dr / 4) * dz)
    per = PI * b["radius"] ** 2 * b["duration"] * b["velocity"] * b["density"] / b["n"]
    return r, per * vol / mean


def _cell(x):
    return torch.clamp(torch.ceil(x).long() - 1, min=0)


def _piece(i, a0, b0, a1, b1):
    """The r-z current of a straight piece inside a cell of row i from offsets
    (a0, b0) to (a1, b1): j_z at (i, k), (i+1, k) in units of q / (4 pi dr^2
    dt) and j_r at (i, k), (i, k+1) in units of q / (2 pi dr dz dt)."""
    da, db, fm, f = a1 - a0, b1 - b0, 0.5 * (a0 + a1), i.double()
    axis = i == 0
    fs = torch.where(axis, torch.ones_like(f), f)
    rm, ro, rn = fs + fm, fs + a0, fs + a1
    s2 = (0.5 * da / rm) ** 2
    eps = torch.zeros_like(s2)
    for m in range(12, 0, -1):
        eps = s2 * (1.0 / (2 * m + 1) + eps)
    ii = fs * (fs + 1)
    z0 = db * ((1 - fm) * (2 * fs + fm) + ii * eps) / (rm * fs)
    z1 = db * (fm * (2 * fs + 1 + fm) - ii * eps) / (rm * (fs + 1))
    q1, q2, q3 = da / (ro * rn), db * da / (2 * rm * rn), db * eps / rm
    r0 = 0.5 * da * (1 - b0) - 0.25 * db * da + 0.5 * ii * (q1 * (1 - b0) - q2 - q3)
    r1 = 0.5 * da * b0 + 0.25 * db * da + 0.5 * ii * (q1 * b0 + q2 + q3)
    half = fs + 0.5
    a = 0.5 * da * (1 - b0) - 0.25 * db * da
    b = 0.5 * da * b0 + 0.25 * db * da
    return (torch.where(axis, 8 * db * (1 - fm), z0), torch.where(axis, db * (1 + fm), z1),
            torch.where(axis, 2 * a, r0 / half), torch.where(axis, 2 * b, r1 / half))


class _Exact:
    """One simulation advanced in FP64."""

    def __init__(self, case, seed):
        self.case, self.g = case, _geometry(case)
        self.pusher = case.get("pusher", "boris")
        g = self.g
        self.f = {k: torch.from_numpy(a).to(DEVICE) for k, a in _fields(case, g, seed).items()}
        self.sigma = torch.from_numpy(_sigma(g)).to(DEVICE)
        self.t, self.parts = 0.0, []
        for q, m, r, z, vr, vphi, vz, w in _plasma(case, g, seed):
            self.parts.append({"q": q * EL_CHARGE, "m": m * EL_MASS, "x": r / g["dr"],
                               "y": z / g["dz"], "v": [vr.clone(), vphi.clone(), vz.clone()],
                               "w": w, "alive": None})
        self.bunch = _bunch(case, g)
        if self.bunch:
            r, w = _bunch_state(self.bunch, g)
            n = self.bunch["n"]
            zero = torch.zeros(n, dtype=torch.float64, device=DEVICE)
            self.parts.append({"q": -EL_CHARGE, "m": EL_MASS,
                               "x": torch.from_numpy(r).to(DEVICE) / g["dr"], "y": zero.clone(),
                               "v": [zero.clone() for _ in range(3)],
                               "w": torch.from_numpy(w).to(DEVICE),
                               "alive": torch.zeros(n, dtype=torch.bool, device=DEVICE)})
            self.places = torch.from_numpy(_radical_inverse(n, 11)).to(DEVICE)

    def _inject(self):
        b, g = self.bunch, self.g
        if not b or not 0.0 <= self.t < b["duration"]:
            return
        per = b["n"] // math.ceil(b["duration"] / g["dt"])
        start = int(self.t / g["dt"] * per)
        sel, p = slice(start, min(start + per, b["n"])), self.parts[-1]
        p["y"][sel] = (b["velocity"] * g["dt"] * self.places[sel] + g["dz"] / 2) / g["dz"]
        p["v"][2][sel] = b["velocity"]
        p["alive"][sel] = True

    def _h(self):
        f, g = self.f, self.g
        dt, dr, dz = g["dt"], g["dr"], g["dz"]
        half = {k: torch.zeros_like(f["H_r"]) for k in ("H_r", "H_phi", "H_z")}
        a = dt * (f["E_phi"][:, 1:] - f["E_phi"][:, :-1]) / (dz * MAGN_CONST)
        half["H_r"][:, :-1] = f["H_r"][:, :-1] + a / 2
        f["H_r"][:, :-1] += a
        c = (slice(0, -1), slice(0, -1))
        b = dt * ((f["E_z"][1:, :-1] - f["E_z"][c]) / dr -
                  (f["E_r"][:-1, 1:] - f["E_r"][c]) / dz) / MAGN_CONST
        half["H_phi"][c] = f["H_phi"][c] + b / 2
        f["H_phi"][c] += b
        i = torch.arange(g["nr"] - 1, dtype=torch.float64, device=DEVICE)[:, None]
        e0, e1 = f["E_phi"][c], f["E_phi"][1:, :-1]
        d = dt * ((e1 + e0) / (2 * dr * (i + 0.5)) + (e1 - e0) / dr) / MAGN_CONST
        half["H_z"][c] = f["H_z"][c] - d / 2
        f["H_z"][c] -= d
        return half

    def _e(self, j):
        f, g = self.f, self.g
        dt, dr, dz = g["dt"], g["dr"], g["dz"]
        st = self.sigma * dt
        ke, kh = (2 * EPSILON0 - st) / (2 * EPSILON0 + st), 2 * dt / (2 * EPSILON0 + st)
        hp, hr, hz = f["H_phi"], f["H_r"], f["H_z"]
        c = (slice(0, -1), slice(1, -1))
        f["E_r"][c] = f["E_r"][c] * ke[c] - (j["J_r"][c] +
                                             (hp[c] - hp[:-1, :-2]) / dz) * kh[c]
        f["E_z"][0, :-1] = (f["E_z"][0, :-1] * ke[0, :-1] -
                            (j["J_z"][0, :-1] - 4 / dr * hp[0, :-1]) * kh[0, :-1])
        c = (slice(1, -1), slice(0, -1))
        i = torch.arange(1, g["nr"] - 1, dtype=torch.float64, device=DEVICE)[:, None]
        f["E_z"][c] = f["E_z"][c] * ke[c] - (j["J_z"][c] - (hp[c] - hp[:-2, :-1]) / dr -
                                             (hp[c] + hp[:-2, :-1]) / (2 * dr * i)) * kh[c]
        c = (slice(1, -1), slice(1, -1))
        f["E_phi"][c] = f["E_phi"][c] * ke[c] - (
            j["J_phi"][c] - (hr[c] - hr[1:-1, :-2]) / dz + (hz[c] - hz[:-2, 1:-1]) / dr) * kh[c]

    def _push(self, q, m, e, h, v):
        """The pushers (src/particles.cpp:1025-1254): velocity to velocity."""
        c1, c2 = q * self.g["dt"] / (2 * m), LIGHT_SPEED ** 2

        def dot(a, b):
            return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

        def cross(a, b):
            return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                    a[0] * b[1] - a[1] * b[0]]

        rel = self.pusher != "boris_classic"
        gm = 1 / torch.sqrt(1 - dot(v, v) / c2) if rel else 1.0
        u = [a * gm for a in v]
        if self.pusher == "vay":
            ee, bb = [a * 2 * c1 for a in e], [a * MAGN_CONST * c1 * 2 * c1 * c1 for a in h]
            k = cross(u, bb)
            gm = 1 / torch.sqrt(1 + dot(u, u) / c2)
            u = [a + b + gm * d for a, b, d in zip(u, ee, k)]
            alpha = 1 + dot(u, u) / c2
            b2 = dot(bb, bb)
            sg, ub = alpha - b2, dot(u, bb)
            alpha = 1 / torch.sqrt(0.5 * (sg + torch.sqrt(sg * sg + 4 * (b2 + ub * ub))))
            bb = [a * alpha for a in bb]
            ub, k = dot(u, bb), cross(u, bb)
            sg = 1 / (1 + dot(bb, bb))
            u = [sg * (a + ub * b + d) for a, b, d in zip(u, bb, k)]
        else:
            um = [a + c1 * b for a, b in zip(u, e)]
            gm = 1 / torch.sqrt(1 + dot(um, um) / c2) if rel else 1.0
            tb = [a * MAGN_CONST * c1 * gm for a in h]
            up = [a + b for a, b in zip(um, cross(um, tb))]
            k = 2 / (1 + dot(tb, tb))
            u = [a + k * b + c1 * d for a, b, d in zip(um, cross(up, tb), e)]
        gm = 1 / torch.sqrt(1 + dot(u, u) / c2) if rel else 1.0
        return [a * gm for a in u]

    def _gather(self, half, x, y):
        nz, f = self.g["nz"], self.f
        ih, i0 = _cell(x - 0.5), _cell(x)
        kh, k0 = _cell(y - 0.5), _cell(y)
        r1, r3 = (x - 0.5) ** 2, (x + 0.5) ** 2
        m = (ih + 1.0) ** 2
        wh = ((m - r1) / (2 * (ih + 1.0)), (r3 - m) / (2 * (ih + 3.0)))
        m = (i0 + 0.5) ** 2
        v0 = torch.where(x > 1, 2.0 * i0, torch.full_like(x, 0.25))
        wn = ((m - r1) / v0, (r3 - m) / (2 * (i0 + 2.0)))
        zh, zn = (kh + 1.5 - y, y - kh - 0.5), (k0 + 1 - y, y - k0)

        def take(a, i, k, wr, wz):
            a, t = a.reshape(-1), i * nz + k
            return (wz[0] * (a[t] * wr[0] + a[t + nz] * wr[1]) +
                    wz[1] * (a[t + 1] * wr[0] + a[t + nz + 1] * wr[1]))

        e = [take(f["E_r"], ih, k0, wh, zn), take(f["E_phi"], i0, k0, wn, zn),
             take(f["E_z"], i0, kh, wn, zh)]
        h = [take(half["H_r"], i0, kh, wn, zh), take(half["H_phi"], ih, kh, wh, zh),
             take(half["H_z"], ih, k0, wh, zn)]
        return e, h

    def _move(self, p, sel, half, j):
        """One chunk of particles through gather, push, moves and deposits."""
        g, nz = self.g, self.g["nz"]
        dt, dr, dz = g["dt"], g["dr"], g["dz"]
        x0, y0, w = p["x"][sel], p["y"][sel], p["w"][sel]
        e, h = self._gather(half, x0, y0)
        v = self._push(p["q"], p["m"], e, h, [a[sel] for a in p["v"]])
        hx, hy, hz = v[0] * dt / (2 * dr), v[1] * dt / (2 * dr), v[2] * dt / (2 * dz)
        x1, y1 = torch.sqrt((x0 + hx) ** 2 + hy * hy), y0 + hz

        def add(grid, i, k, val):
            j[grid].reshape(-1).index_add_(0, i * nz + k, val)

        i, k = _cell(x1), _cell(y1)
        a, b = x1 - i, y1 - k
        low = torch.where(i >= 1, 2.0 * i, torch.full_like(x1, 0.25))
        cur = p["q"] * w * v[1] / (2 * PI * dz * dr * dr)
        wa, wb = (1 - a) * (2 * i + a) / (x1 * low), a * (2 * i + 1 + a) / (x1 * 2 * (i + 1))
        for s, t, val in ((0, 0, (1 - b) * wa), (1, 0, (1 - b) * wb), (0, 1, b * wa),
                          (1, 1, b * wb)):
            add("J_phi", i + s, k + t, cur * val)
        x, y = x1 + hx, y1 + hz
        wr, wz = g["nr"] - 1.5, g["nz"] - 1.5
        alive = torch.ones_like(x, dtype=torch.bool)
        if p["alive"] is None:
            v[0], x = torch.where(x > wr, -v[0], v[0]), torch.where(x > wr, 2 * wr - x, x)
            v[2], y = torch.where(y > wz, -v[2], v[2]), torch.where(y > wz, 2 * wz - y, y)
        else:
            alive = (x <= wr) & (y <= wz)
        v[0], x = torch.where(x < 0.5, -v[0], v[0]), torch.where(x < 0.5, 1 - x, x)
        v[2], y = torch.where(y < 0.5, -v[2], v[2]), torch.where(y < 0.5, 1 - y, y)
        rn = torch.sqrt(x * x + hy * hy)
        i0, k0 = _cell(x0), _cell(y0)
        # face crossings along the path, each as a share of it
        i2, k2 = _cell(rn), _cell(y)
        far = torch.full_like(x0, 2.0)
        tr = torch.where(i2 == i0, far, (torch.maximum(i0, i2) - x0) / (rn - x0))
        tz = torch.where(k2 == k0, far, (torch.maximum(k0, k2) - y0) / (y - y0))
        ts = [torch.zeros_like(x0), torch.clamp(torch.minimum(tr, tz), max=1.0),
              torch.clamp(torch.maximum(tr, tz), max=1.0), torch.ones_like(x0)]
        cz, cr = p["q"] / (4 * PI * dr * dr * dt), p["q"] / (2 * PI * dr * dz * dt)
        for n in range(3):
            on = alive & (ts[n + 1] > ts[n])
            if n:
                on = on.nonzero()[:, 0]
                if not on.numel():
                    continue
            t0, t1 = ts[n][on], ts[n + 1][on]
            xs, ys, dx, dy = x0[on], y0[on], (rn - x0)[on], (y - y0)[on]
            ci = torch.floor(xs + 0.5 * (t0 + t1) * dx).long()
            ck = torch.floor(ys + 0.5 * (t0 + t1) * dy).long()
            bi, bk = xs - ci, ys - ck
            z0, z1, r0, r1 = _piece(ci, bi + t0 * dx, bk + t0 * dy, bi + t1 * dx, bk + t1 * dy)
            ws = w[on]
            add("J_z", ci, ck, cz * ws * z0)
            add("J_z", ci + 1, ck, cz * ws * z1)
            add("J_r", ci, ck, cr * ws * r0)
            add("J_r", ci, ck + 1, cr * ws * r1)
        sn = hy / rn
        cs = torch.sqrt(1 - sn * sn)
        turn = [cs * v[0] - sn * v[1], sn * v[0] + cs * v[1]]
        p["v"][0][sel] = torch.where(alive, turn[0], v[0])
        p["v"][1][sel] = torch.where(alive, turn[1], v[1])
        p["v"][2][sel], p["x"][sel], p["y"][sel] = v[2], rn, y
        if p["alive"] is not None:
            p["alive"][sel] = alive

    def step(self):
        self._inject()
        half = self._h()
        self.j = j = {k: torch.zeros_like(self.f["E_r"]) for k in ("J_r", "J_phi", "J_z")}
        for p in self.parts:
            if p["alive"] is not None:
                live = p["alive"].nonzero()[:, 0]
                if live.numel():
                    self._move(p, live, half, j)
                continue
            for s in range(0, p["x"].numel(), 1 << 22):
                self._move(p, slice(s, min(s + (1 << 22), p["x"].numel())), half, j)
        self._e(j)
        self.t += self.g["dt"]

    def species(self, s):
        p = self.parts[s]
        return dict(zip(PARTICLE, (p["x"] * self.g["dr"], p["y"] * self.g["dz"], *p["v"])))


def _weighting(g, x, y, amount, low, out):
    """amount of each particle over the four nodes around it, by the volumes of
    the ring pieces that it overlaps (src/particles.cpp:101-226), per node
    volume; `low` (the axis row's volume in pi dz dr^2) as both weightings."""
    i, k = _cell(x), _cell(y)
    inner = x <= 0.5
    r1, m, r3 = (x - 0.5) ** 2, (i + 0.5) ** 2, (x + 0.5) ** 2
    own = torch.where(inner, 2 * x * x + 0.5, 2 * x)  # the particle's volume / (pi dz dr^2)
    a = torch.where(inner, 0.5 - x + x * x, m - r1) / own
    b = (r3 - m) / own
    va = torch.where(i >= 1, 2.0 * i, torch.full_like(x, low))
    z1, z2 = k + 1 - y, y - k
    scale = amount / (PI * g["dz"] * g["dr"] ** 2)
    for s, t, val in ((0, 0, z1 * a / va), (1, 0, z1 * b / (2 * (i + 1.0))), (0, 1, z2 * a / va),
                      (1, 1, z2 * b / (2 * (i + 1.0)))):
        out.reshape(-1).index_add_(0, (i + s) * g["nz"] + k + t, scale * val)


def _exact_dump(case, seed):
    g = _geometry(case)
    el, ion = _plasma(case, g, seed)
    x, y, v, w = el[2] / g["dr"], el[3] / g["dz"], list(el[4:7]), el[7]
    zero = torch.zeros((g["nr"], g["nz"]), dtype=torch.float64, device=DEVICE)
    grid = {k: zero.clone() for k in ("rho_electrons", "density", "density_ions")}
    _weighting(g, x, y, -EL_CHARGE * w, 0.25, grid["rho_electrons"])
    _weighting(g, x, y, w, 0.25, grid["density"])
    _weighting(g, x, y, ION_MASS * w, 0.25, grid["density_ions"])
    sums = torch.zeros((5, g["nr"] * g["nz"]), dtype=torch.float64, device=DEVICE)
    t = _cell(x) * g["nz"] + _cell(y)
    v2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
    for row, val in zip(sums, (torch.sqrt(v2), *v, torch.ones_like(x))):
        row.index_add_(0, t, val)
    sq = (sums[0] ** 2 - sums[1] ** 2 - sums[2] ** 2 - sums[3] ** 2) / sums[4] ** 2
    temp = (EL_MASS * sq / 2 / EL_CHARGE).reshape(g["nr"], g["nz"])
    temp[-1], temp[:, -1] = 0.0, 0.0
    f = {k: torch.from_numpy(a).to(DEVICE) for k, a in _fields(case, g, seed).items()}
    i = torch.arange(g["nr"], dtype=torch.float64, device=DEVICE)[:, None]
    vol = torch.where(i == 0, 0.25 * torch.ones_like(i), 2 * i) * PI * g["dz"] * g["dr"] ** 2
    e2 = sum(f[k] ** 2 for k in GRIDS[:3])
    h2 = sum(f[k] ** 2 for k in GRIDS[3:6])
    b2 = v2 / LIGHT_SPEED ** 2
    sq = torch.sqrt(1 - b2)
    kin = (EL_MASS * w * LIGHT_SPEED ** 2 * b2 / (sq * (1 + sq))).sum()
    return {"rho_electrons": grid["rho_electrons"], "rho_ions": -grid["rho_electrons"],
            "temperature": temp,
            "density": grid["density"], "density_ions": grid["density_ions"],
            "E_z": f["E_z"].reshape(-1),
            "field_energy": float((0.5 * (EPSILON0 * e2 + MAGN_CONST * h2) * vol).sum()),
            "kinetic_energy": float(kin), "rho_norm": None, "alive": None}


def _exact_poisson(case, seed):
    """Sine transform along z as a matrix product, the radial equation of each
    mode by elimination, and the transform back (src/poissonDirichlet.cpp:23-98)."""
    g = _geometry(case)
    nr, nz, dr, dz = g["nr"], g["nz"], g["dr"], g["dz"]
    rho = torch.from_numpy(_rho(g, seed)).to(DEVICE)
    n = torch.arange(1, nz + 1, device=DEVICE)
    turn = (n[:, None] * n[None, :] % (2 * (nz + 1))).double()  # the angle, reduced in whole numbers
    sine = torch.sin(turn * PI / (nz + 1))
    t = dr * dr / EPSILON0 * (rho @ sine)
    b = 2 * (1 - dr * dr / (dz * dz) * (torch.cos(n.double() * PI / (nz + 1)) - 1))
    al, be = [4 / (2 + b)], [t[0] / (2 + b)]
    for i in range(1, nr - 1):
        a, c = 1 - 1 / (2 * i), 1 + 1 / (2 * i)
        den = b - al[-1] * a
        be.append((t[i] + be[-1] * a) / den)
        al.append(c / den)
    fi = torch.zeros_like(rho)
    for i in range(nr - 2, -1, -1):
        fi[i] = be[i] + al[i] * fi[i + 1]
    fi = (fi @ sine) * 2 / (nz + 1)
    er, ez = torch.zeros_like(fi), torch.zeros_like(fi)
    er[:-1], ez[:, :-1] = (fi[:-1] - fi[1:]) / dr, (fi[:, :-1] - fi[:, 1:]) / dz
    return {"phi": fi, "E_r": er, "E_z": ez}


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        return _exact_poisson(case, seed)
    if kind == "dump":
        return _exact_dump(case, seed)
    if kind == "adjoint":
        # the gradient holds, beside the derivative of each trajectory, an
        # estimate of the jumps that many particles cross: no plain value
        return None
    if work(dict(case))["flops"] > 400 * 5e8:
        return None  # over twenty seconds
    if kind == "ensemble":
        out = []
        for c, s in _ensemble_cases(case, seed):
            ex = _Exact(c, s)
            for _ in range(case["steps"]):
                ex.step()
            out.append({"E_r": ex.f["E_r"], "E_z": ex.f["E_z"], "J_z": ex.j["J_z"]})
        return out
    ex = _Exact(case, seed)
    for _ in range(case["steps"]):
        ex.step()
    every = range(len(ex.parts))
    if kind == "host_loop":
        return {"species": [dict(ex.species(s), alive=None) for s in every], "E_z": ex.f["E_z"]}
    out = {k: ex.f[k] if k[0] != "J" else ex.j[k] for k in GRIDS}
    if case["cells_r"] * case["cells_z"] * case["ppc"] <= 10000 and not case["sort"]:
        for s in every:
            out["species%d" % s] = ex.species(s)
            out["alive%d" % s] = None
    return out
