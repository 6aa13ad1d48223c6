"""What the engine's users have it do, as measurable cases: one pass of each
goes through the package's public entry points, with inputs made from a seed.

The sizes are those of the configurations this repository is built around
(10,000 and 2^20 electron bulk runs, the 64-ensemble velocity-field sweep, the
201 x 101 resistor, the eight-bias 401 x 201 MOSFET batch), and generic ones
beside them: single-step calls, odd and ragged sizes, larger Poisson grids.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import viennaemc_gb300 as emc
from viennaemc_gb300 import _lib as clib
from viennaemc_gb300 import device as dev2d
from viennaemc_gb300 import p2p, physics

Q, KB, EPS0 = 1.60219e-19, 1.38066e-23, 8.85419e-12  # the physical constants of the models
DIRS = {"100": (1, 0, 0), "111": (1, 1, 1)}
SCHEMES = {"ngp": dev2d.NGP, "cic": dev2d.CIC, "nec": dev2d.NEC}


def listed():
    return [
        # the reference's own loop: one moveParticles(dt) per call with its averages read
        # back, on the 10,000-electron ensemble, in the handler's default precision
        {"name": "handler_step_10k_fp64", "kind": "handler", "precision": "fp64", "n": 10000,
         "field": 1e5, "dir": "100", "T": 300.0, "box": 1e-6},
        # the small bulk run in the parity precision: 100 steps, observables and the
        # electrons themselves
        {"name": "bulk_10k_fp64", "kind": "bulk", "precision": "fp64", "n": 10000, "steps": 100,
         "field": 1e5, "dir": "100", "T": 300.0, "state": True, "grain": False},
        # a larger parity run at a low temperature, the field along <111>
        {"name": "bulk_250k_fp64", "kind": "bulk", "precision": "fp64", "n": 250007, "steps": 20,
         "field": 1e6, "dir": "111", "T": 77.0, "state": False, "grain": False},
        # the headline run: 2^20 electrons at 1e6 V/m, 20 steps with their observables
        {"name": "bulk_1M_fp32", "kind": "bulk", "precision": "fp32", "n": 1 << 20, "steps": 20,
         "field": 1e6, "dir": "100", "T": 300.0, "state": False, "grain": False},
        # the velocity-field sweep: 64 uneven ensembles, four temperatures, graph replay
        {"name": "sweep_64_fp32", "kind": "sweep", "precision": "fp32", "ensembles": 64,
         "lo": 1e4, "hi": 1e6, "steps": 20, "layout": 2024},
        # the particle-particle sums of the FMM handlers, host arrays in and out
        {"name": "p2p_32k_fp32", "kind": "p2p", "precision": "fp32", "n": 32768, "images": 0,
         "cutoff": 1e9},
        # bulk steps with those sums in every step (the FMM bulk handler, as it comes)
        {"name": "fmm_steps_fp64", "kind": "fmm", "precision": "fp64", "n": 5001, "steps": 3,
         "images": 0},
        # the resistor: 5e5 electrons, Poisson, field, move, contacts, CIC, ten steps
        {"name": "resistor_201x101_fp32", "kind": "resistor", "precision": "fp32", "nx": 201,
         "ny": 101, "h": 0.5e-9, "electrons": 5e5, "scheme": "cic", "steps": 10},
        # a small resistor in the simulation's default precision, nearest-node scheme
        {"name": "resistor_101x51_fp64", "kind": "resistor", "precision": "fp64", "nx": 101,
         "ny": 51, "h": 1e-9, "electrons": 5e4, "scheme": "ngp", "steps": 5},
        # the MOSFET's drain sweep: eight uneven simulations stepped together
        {"name": "mosfet_8x401x201_fp32", "kind": "mosfet", "precision": "fp32", "engines": 8,
         "nx": 401, "ny": 201, "lo": 2e5, "hi": 6e5, "steps": 5, "layout": 5},
        # the solver as a plugin of the host's own loop: potential and concentration in,
        # potential out, on a grid above those of the configurations
        {"name": "poisson_801x401", "kind": "poisson", "shape": "resistor", "nx": 801, "ny": 401,
         "equilibrium": False, "fp32": True, "noalloc": False},
        # the solve that allocates nothing, on the caller's device arrays
        {"name": "noalloc_201x101", "kind": "poisson", "shape": "resistor", "nx": 201, "ny": 101,
         "equilibrium": False, "fp32": True, "noalloc": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["handler", "bulk", "bulk", "bulk", "sweep", "p2p", "p2p", "fmm",
                       "resistor", "resistor", "mosfet", "poisson", "poisson", "poisson"])
    prec = rng.choice(["fp32", "fp64"])
    if kind == "handler":
        return {"kind": kind, "precision": prec, "n": round(_log(rng, 1000, 60000)),
                "field": _log(rng, 1e4, 1e7), "dir": rng.choice(list(DIRS)),
                "T": rng.choice([77.0, 200.0, 300.0, 400.0]), "box": 1e-6}
    if kind == "bulk":
        n = round(_log(rng, 1000, 1 << 20 if prec == "fp32" else 250000))
        most = min(400.0, (2.1e7 if prec == "fp32" else 4e6) / n)
        return {"kind": kind, "precision": prec, "n": n, "steps": round(_log(rng, 1, max(most, 2))),
                "field": _log(rng, 1e4, 1e7), "dir": rng.choice(list(DIRS)),
                "T": rng.choice([77.0, 200.0, 300.0, 400.0]), "state": n < 30000,
                "grain": rng.random() < 0.2}
    if kind == "sweep":
        e = rng.randint(3, 64)
        return {"kind": kind, "precision": prec, "ensembles": e, "lo": 1e3,
                "hi": 3e5 if prec == "fp32" else 2e4, "steps": rng.randint(1, 20),
                "layout": rng.randrange(1 << 20)}
    if kind == "p2p":
        images = 1 if rng.random() < 0.25 else 0
        top = (32768 if prec == "fp32" else 12000) / (5 if images else 1)
        return {"kind": kind, "precision": prec, "n": round(_log(rng, 300, top)),
                "images": images, "cutoff": rng.choice([1e9, 1e9, 0.0])}
    if kind == "fmm":
        images = 1 if rng.random() < 0.25 else 0
        return {"kind": kind, "precision": prec, "n": round(_log(rng, 300, 1000 if images else 5000)),
                "steps": rng.randint(1, 3), "images": images}
    if kind == "resistor":
        nx, ny = round(_log(rng, 41, 201)), round(_log(rng, 31, 101))
        return {"kind": kind, "precision": prec, "nx": nx, "ny": ny,
                "h": rng.choice([0.5e-9, 1e-9]),
                "electrons": round(_log(rng, 1e4, 5e5 if prec == "fp32" else 6e4)),
                "scheme": rng.choice(list(SCHEMES)), "steps": rng.randint(1, 10)}
    if kind == "mosfet":
        return {"kind": kind, "precision": "fp32", "engines": rng.randint(1, 8),
                "nx": rng.randint(101, 401), "ny": rng.randint(81, 201), "lo": 1e5, "hi": 6e5,
                "steps": rng.randint(1, 5), "layout": rng.randrange(1 << 20)}
    noalloc = rng.random() < 0.4
    top = 131072 if noalloc else 801 * 401
    nx = round(_log(rng, 41, 801))
    ny = round(_log(rng, 31, min(401, top // nx)))
    # a step of a running bar, or a MOSFET's equilibrium from its neutral potential
    shape = rng.choice(["resistor", "resistor", "mosfet"])
    return {"kind": "poisson", "shape": shape, "nx": nx, "ny": ny,
            "equilibrium": shape == "mosfet",
            "fp32": noalloc or nx * ny > 80601 or rng.random() < 0.7, "noalloc": noalloc}


# ---- models and devices ----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _silicon(T, grain=False):
    return emc.silicon_electron("jacoboni", temperature=T, n_levels=3000, max_energy=3.0,
                                grain=(0.5, 1e13) if grain else None)


def _resistor(nx, ny, h, electrons):
    """n+ silicon bar, ohmic contacts with 0.5 V across its length."""
    lx, ly = (nx - 1) * h, (ny - 1) * h
    dev = dev2d.Device(physics.silicon_material(), (lx, ly), (h, h))
    dev.setDeviceWidth(electrons / (1e24 * lx * ly))
    dev.addConstantDopingRegion((0, 0), (lx, ly), 1e24)
    dev.addOhmicContact(dev2d.XMAX, 0.0, (0,), (ly,))
    dev.addOhmicContact(dev2d.XMIN, 0.5, (0,), (ly,))
    return dev


def _mosfet(nx, ny, vds, electrons=3.9e5):
    """n-MOSFET at 0.5 nm: source and drain 1e26 to a fifth of the depth, gate over the
    middle quarter behind 1 nm of oxide, substrate contact at the back."""
    h = 0.5e-9
    lx, ly = (nx - 1) * h, (ny - 1) * h
    a, b = (round(f * (nx - 1)) * h for f in (0.375, 0.625))
    d = round(0.2 * (ny - 1)) * h
    dev = dev2d.Device(physics.silicon_material(), (lx, ly), (h, h))
    dev.setDeviceWidth(electrons / (1e26 * (lx - (b - a)) * d))
    dev.addConstantDopingRegion((0, d), (lx, ly), -1e24)
    dev.addConstantDopingRegion((0, 0), (a, d), 1e26)
    dev.addConstantDopingRegion((a, 0), (b, d), -1e24)
    dev.addConstantDopingRegion((b, 0), (lx, d), 1e26)
    dev.addOhmicContact(dev2d.YMAX, 0.0, (0,), (lx,))
    dev.addOhmicContact(dev2d.YMIN, 0.0, (0,), (a,))
    dev.addGateContact(dev2d.YMIN, 1.0, (a,), (b,), 3.9, 1e-9, 1.12 / 2)
    dev.addOhmicContact(dev2d.YMIN, vds, (b,), (lx,))
    return dev


def _device_electrons(dev, first_order):
    return physics.silicon_electron("refbulk", n_levels=1000, max_energy=4.0,
                                    regions=list(range(dev.n_regions)), coulomb=True,
                                    region_doping=dev.getDopingRegionDoping,
                                    first_order=first_order)


def _spec(model, n, case, seed, T):
    return emc.EnsembleSpec(model, n, case["field"], DIRS[case["dir"]], (1e-6,) * 3, 1e-15, seed,
                            0, T)


def _charges(case, seed):
    """Electrons and donors, alternating, uniform in a 100 nm cube."""
    rs = np.random.default_rng(seed)
    n = case["n"]
    return rs.random((3, n)) * 1e-7, np.where(np.arange(n) % 2 == 0, -Q, Q)


def _sweep_layout(case):
    rs = np.random.default_rng(case["layout"])
    out = []
    for e in range(case["ensembles"]):
        out.append((e // 8 % 4, int(round(math.exp(rs.uniform(math.log(case["lo"]),
                                                              math.log(case["hi"]))))),
                    float(np.logspace(4, 7, 8)[e % 8]), "100" if e < 32 else "111"))
    return out


def _mosfet_layout(case):
    rs = np.random.default_rng(case["layout"])
    k = case["engines"]
    return [(float(v), float(rs.uniform(case["lo"], case["hi"])))
            for v in np.linspace(0.0, 1.0, k)]


def _grids(case, seed):
    """The device, a starting potential and a noisy electron concentration: those of the
    neutral device, as a running bar's next step or a MOSFET's first solve finds them."""
    nx, ny = case["nx"], case["ny"]
    dev = _resistor(nx, ny, 0.5e-9, 5e5) if case["shape"] == "resistor" else \
        _mosfet(nx, ny, 0.05)
    rs = np.random.default_rng(seed)
    c = dev.doping / dev.material.Ni
    pot = np.arcsinh(0.5 * c)
    per = 60.0  # superparticles at a node of full doping
    n = np.exp(pot)
    full = max(float(n.max()), 1.0)
    conc = rs.poisson(per * n / full) * (full / per)
    if case["shape"] == "resistor":  # the applied voltage falls along the bar
        pot = pot + np.tile(np.linspace(0.5, 0.0, nx) / dev.getThermalVoltage(), ny)
        pot = pot + 0.02 * rs.standard_normal(pot.size)
    else:
        pot = pot + 0.02 * rs.standard_normal()
    return dev, pot, (None if case["equilibrium"] else conc)


# ---- the cases -------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "handler":
        h = emc.BulkParticleHandler((case["box"],) * 3, _silicon(case["T"]), DIRS[case["dir"]],
                                    case["field"], seed=seed + 1, temperature=case["T"],
                                    precision=case["precision"], dt=1e-15)
        h.generateInitialParticles(n=case["n"])
        s["handler"] = h
    elif kind == "bulk":
        s["batch"] = emc.BulkBatch([_silicon(case["T"], case["grain"])],
                                   [_spec(0, case["n"], case, seed + 1, case["T"])],
                                   case["precision"])
        s["batch"].init_particles(0)
    elif kind == "sweep":
        temps = (77.0, 200.0, 300.0, 400.0)
        specs = [_spec(m, n, {"field": f, "dir": d}, seed + 1 + 1000 * e, temps[m])
                 for e, (m, n, f, d) in enumerate(_sweep_layout(case))]
        b = emc.BulkBatch([_silicon(T) for T in temps], specs, case["precision"])
        for e in range(len(specs)):
            b.init_particles(e)
        b.set_graph(True)
        s["batch"] = b
    elif kind == "p2p":
        s["pos"], s["q"] = _charges(case, seed)
    elif kind == "fmm":
        h = emc.FMMBulkParticleHandler((1e-7,) * 3, _silicon(300.0), (1, 0, 0), 1e6,
                                       images=case["images"], seed=seed + 1,
                                       precision=case["precision"], dt=1e-16)
        h.generateInitialParticles(n=case["n"], doping=0.0)
        s["handler"] = h
    elif kind == "resistor":
        dev = _resistor(case["nx"], case["ny"], case["h"], case["electrons"])
        sim = dev2d.DeviceSimulation(dev, _device_electrons(dev, True),
                                     scheme=SCHEMES[case["scheme"]], dt=1e-16, seed=seed + 1,
                                     precision=case["precision"])
        sim.calcEquilibriumCharacteristics()
        s["sims"] = [sim]
    elif kind == "mosfet":
        s["sims"] = []
        for k, (vds, count) in enumerate(_mosfet_layout(case)):
            dev = _mosfet(case["nx"], case["ny"], vds, count)
            sim = dev2d.DeviceSimulation(dev, _device_electrons(dev, False), scheme=dev2d.CIC,
                                         dt=1e-16, seed=seed + 1 + 1000 * k,
                                         precision=case["precision"], poisson_max_cycles=200,
                                         tau_region_is_valley=True)
            sim.calcEquilibriumCharacteristics()
            s["sims"].append(sim)
    else:
        dev, pot, conc = _grids(case, seed)
        s["pot"], s["conc"] = pot, conc
        if case["noalloc"]:
            s["dev"], s["desc"] = dev, dev.desc()
            s["d_start"] = torch.tensor(pot, device="cuda")
            s["d_pot"] = torch.empty_like(s["d_start"])
            s["d_conc"] = None if conc is None else torch.tensor(conc, device="cuda")
        else:
            s["sim"] = dev2d.DeviceSimulation(dev, _device_electrons(dev, False),
                                              capacity=4096, poisson_max_cycles=200,
                                              poisson_fp32=case["fp32"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "handler":
        return dict(s["handler"].moveParticles(1e-15))
    if kind in ("bulk", "sweep"):
        b = s["batch"]
        out = emc.BulkBatch.averages(b.step(case["steps"]), [sp.n_particles for sp in b.specs])
        if case.get("state"):
            st = b.get_state(0)
            out["electrons"] = {f: getattr(st, f) for f in ("kx", "ky", "kz", "px", "py", "pz",
                                                            "energy", "tau", "valley", "sub")}
        return out
    if kind == "p2p":
        return p2p.coulomb(s["pos"], s["q"], case["cutoff"], 1e-7, case["images"],
                           case["precision"])
    if kind == "fmm":
        h = s["handler"]
        out = dict(h.moveParticles(1e-16, case["steps"]))
        out["force"], out["potential"] = h.getCoulomb()
        return out
    if kind in ("resistor", "mosfet"):
        if len(s["sims"]) == 1:
            netto = [s["sims"][0].performEMCStep(case["steps"])]
        else:
            netto = dev2d.DeviceSimulation.performEMCStepMany(s["sims"], case["steps"])
        return [{"netto": n, "potential": sim.potential, "concentration": sim.concentration}
                for n, sim in zip(netto, s["sims"])]
    if case["noalloc"]:
        s["d_pot"].copy_(s["d_start"])
        rel, cyc = ctypes.c_double(), ctypes.c_int32()
        clib.check(clib.lib().emcg_poisson_solve_noalloc(
            ctypes.byref(s["desc"]), ctypes.c_void_p(s["d_pot"].data_ptr()),
            None if s["d_conc"] is None else ctypes.c_void_p(s["d_conc"].data_ptr()), 1, 0, 1e-8,
            200, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(rel),
            ctypes.byref(cyc)))
        return s["d_pot"]
    sim = s["sim"]
    sim.set_grid(clib.GRID_POTENTIAL, s["pot"])
    if s["conc"] is not None:
        sim.set_grid(clib.GRID_CONC, s["conc"])
    sim.poisson(equilibrium=case["equilibrium"], reset_bc=True)
    return sim.potential


def work(case):
    """Bytes: the electrons' state in and out of the call's launches once, the grids of
    every step once; operations: a free flight of about 60 per electron and step, 20 per
    Coulomb pair, multigrid sweeps of about 600 per node and solve."""
    kind = case["kind"]
    state = 152 if case.get("precision") == "fp64" else 80  # read and written
    if kind == "handler":
        return {"bytes": case["n"] * state + 24, "flops": case["n"] * 60}
    if kind in ("bulk", "sweep"):
        ns = [case["n"]] if kind == "bulk" else [e[1] for e in _sweep_layout(case)]
        b = sum(ns) * state + len(ns) * case["steps"] * 24
        return {"bytes": b + (case["n"] * 84 if case.get("state") else 0),
                "flops": sum(ns) * case["steps"] * 60}
    if kind == "p2p":
        n, boxes = case["n"], (2 * case["images"] + 1) ** 3
        return {"bytes": n * 64, "flops": 20.0 * n * n * boxes}
    if kind == "fmm":
        n, boxes = case["n"], (2 * case["images"] + 1) ** 3
        return {"bytes": case["steps"] * n * (state + 64),
                "flops": case["steps"] * (20.0 * n * 2 * n * boxes + 60.0 * n)}
    if kind in ("resistor", "mosfet"):
        n = case["electrons"] if kind == "resistor" else sum(c for _, c in _mosfet_layout(case))
        nodes = case["nx"] * case["ny"] * (1 if kind == "resistor" else case["engines"])
        return {"bytes": case["steps"] * (n * (state - 8) + nodes * 40),
                "flops": case["steps"] * (n * 80.0 + nodes * 600.0)}
    nodes = case["nx"] * case["ny"]
    return {"bytes": nodes * (16 if case["equilibrium"] else 24), "flops": nodes * 600.0}


# ---- the same in 64 bits ---------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "p2p":
        return _exact_p2p(case, seed)
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    return None  # a Monte Carlo path: each number follows from all random draws before it


def _exact_p2p(case, seed):
    pos, q = _charges(case, seed)
    where = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(pos, device=where)
    c = torch.tensor(q, device=where)
    n, w = case["n"], case["images"]
    force, pot = torch.zeros((3, n), dtype=x.dtype, device=where), torch.zeros_like(c)
    chunk = max(1, (1 << 25) // n)
    for o in [(a, b, d) for a in range(-w, w + 1) for b in range(-w, w + 1)
              for d in range(-w, w + 1)]:
        y = x + 1e-7 * torch.tensor(o, dtype=x.dtype, device=where)[:, None]
        for i in range(0, n, chunk):
            m = min(chunk, n - i)
            d = [x[k, i:i + m, None] - y[k, None, :] for k in range(3)]
            inv = torch.rsqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
            if o == (0, 0, 0):
                inv[torch.arange(m, device=where), torch.arange(i, i + m, device=where)] = 0.0
            # closer than the cutoff radius a pair is moved apart to it
            near = torch.clamp(inv, max=case["cutoff"]) if case["cutoff"] > 0 else inv
            pot[i:i + m] += near @ c
            f = inv * near * near * c[None, :]
            for k in range(3):
                force[k, i:i + m] -= c[i:i + m] * (d[k] * f).sum(1)
    return force.cpu().numpy(), pot.cpu().numpy()


def _exact_poisson(case, seed):
    """Newton's method with conjugate gradients on the finite-difference equation."""
    dev, pot, conc = _grids(case, seed)
    nx, ny, Vt = dev.nx, dev.ny, KB / Q * dev.temperature
    Ni, epsr = dev.material.Ni, dev.material.epsR
    debye = math.sqrt(EPS0 * epsr * Vt / Q / Ni)
    h = [s / debye for s in dev.spacing]
    hF = (h[1] / h[0], h[0] / h[1])
    hP = h[0] * h[1]
    C = (dev.doping / Ni).reshape(ny, nx)
    phi = pot.reshape(ny, nx).copy()
    fixed = np.zeros((ny, nx), bool)
    gs, gv = np.zeros((ny, nx)), np.zeros((ny, nx))
    edges = [(slice(None), 0), (slice(None), nx - 1), (0, slice(None)), (ny - 1, slice(None))]
    for b, at in enumerate(edges):
        for ci, (ctype, volt, par) in enumerate(dev.contacts):
            on = dev.bnd[b] == ci
            v = 0.0 if case["equilibrium"] else volt / Vt
            if ctype == dev2d.OHMIC:
                fixed[at] |= on
                phi[at] = np.where(on, v + np.arcsinh(0.5 * C[at]), phi[at])
            else:
                G = 2 * (par[0] / epsr) / (par[1] / debye) * hF[b // 2] * h[b // 2]
                gs[at] += on * G
                gv[at] += on * G * (par[2] / Vt + v)
    area = np.ones((ny, nx))
    area[:, [0, -1]] *= 0.5
    area[[0, -1], :] *= 0.5
    where = "cuda" if torch.cuda.is_available() else "cpu"
    C, phi, gs, gv, area = (torch.tensor(a, device=where) for a in (C, phi, gs, gv, area))
    free = torch.tensor(~fixed, device=where).to(phi.dtype)
    n_el = None if conc is None else torch.tensor(conc.reshape(ny, nx), device=where)

    def laplace(u):
        v = -2.0 * (hF[0] + hF[1]) * u
        v[:, 1:-1] += hF[0] * (u[:, :-2] + u[:, 2:])
        v[:, 0] += hF[0] * 2 * u[:, 1]
        v[:, -1] += hF[0] * 2 * u[:, -2]
        v[1:-1] += hF[1] * (u[:-2] + u[2:])
        v[0] += hF[1] * 2 * u[1]
        v[-1] += hF[1] * 2 * u[-2]
        return v

    for _ in range(40):
        p = torch.exp(-phi)
        n = torch.exp(phi) if n_el is None else n_el
        react = hP * (p + n if n_el is None else p) + gs
        r = free * area * (laplace(phi) + hP * (p - n + C) + gv - gs * phi)
        diag = area * (2.0 * (hF[0] + hF[1]) + react)
        d = torch.zeros_like(phi)
        z = free * r / diag
        s, rz = z.clone(), (r * z).sum()
        goal = 1e-28 * rz
        for k in range(20000):
            As = free * area * (react * s - laplace(s))
            a = rz / (s * As).sum()
            d += a * s
            r -= a * As
            z = free * r / diag
            new = (r * z).sum()
            s = z + (new / rz) * s
            rz = new
            if k % 50 == 49 and not bool(rz > goal):
                break
        step = torch.clamp(d, -2.0, 2.0)
        phi = phi + step
        if float(step.abs().max()) < 1e-12 * float(phi.abs().max()):
            break
    out = phi.reshape(-1)
    return out if case["noalloc"] else out.cpu().numpy()
