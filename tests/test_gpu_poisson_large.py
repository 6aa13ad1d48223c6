"""Grids whose hierarchy does not fit in one cluster (the finest levels one launch
per phase, the rest in one cluster launch) against one launch per phase
throughout, and the no-allocation solve on such grids and with more coefficient
tuples than its class table holds against the allocating one.  Every form
evaluates the same expressions on the same values, so the first pair agrees to
the rounding that other launches of the same arithmetic may have (1e-13, as the
cluster and multi-launch forms of the configuration grids); the second pair
builds its levels differently (1e-8 of the same target, as test_zz_no_alloc)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bar(nx, ny, gates=0):
    from viennaemc_gb300 import device as D
    from viennaemc_gb300.physics import silicon_material
    h = 0.5e-9
    lx, ly = (nx - 1) * h, (ny - 1) * h
    dev = D.Device(silicon_material(), (lx, ly), (h, h))
    dev.addConstantDopingRegion((0, 0), (lx, ly), 1e24)
    dev.addOhmicContact(D.XMAX, 0.0, (0,), (ly,))
    dev.addOhmicContact(D.XMIN, 0.3, (0,), (ly,))
    for g in range(gates):  # each a coupling of its own
        dev.addGateContact(D.YMIN, 0.1, ((4 * g + 4) * h,), ((4 * g + 6) * h,), 3.9,
                           (1 + 0.01 * g) * 1e-9, 0.5)
    return dev


def _start(dev, seed):
    rs = np.random.default_rng(seed)
    pot = np.arcsinh(0.5 * dev.doping / dev.material.Ni) + 0.02 * rs.standard_normal(dev.nx * dev.ny)
    return pot, rs.poisson(60.0, dev.nx * dev.ny) * (1e24 / dev.material.Ni / 60.0)


def _sim(engine, dev, fp32, rtol=1e-10):
    from viennaemc_gb300 import device as D
    pt = engine.physics.silicon_electron("refbulk", n_levels=100, max_energy=4.0)
    return D.DeviceSimulation(dev, pt, capacity=64, poisson_rtol=rtol, poisson_max_cycles=200,
                              poisson_fp32=fp32)


def _solve(sim, pot, conc):
    from viennaemc_gb300 import _lib as L
    sim.set_grid(L.GRID_POTENTIAL, pot)
    sim.set_grid(L.GRID_CONC, conc)
    info = sim.poisson(equilibrium=False, reset_bc=True)
    return sim.potential, info


@pytest.mark.parametrize("nx,ny,fp32", [(601, 301, True), (1203, 137, True), (399, 398, False)])
def test_tail_in_a_cluster_equals_one_launch_per_phase(engine, nx, ny, fp32):
    dev = _bar(nx, ny)
    pot, conc = _start(dev, nx)
    sim = _sim(engine, dev, fp32)
    assert sim.poisson_mode(-1) == 0  # no cluster holds the whole hierarchy
    a, ia = _solve(sim, pot, conc)
    sim.poisson_mode(0)
    b, ib = _solve(sim, pot, conc)
    sim.close()
    assert ia[1] == ib[1] and ia[0] <= 1e-10
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))


@pytest.mark.parametrize("nx,ny,gates", [(201, 101, 0), (360, 361, 0), (301, 61, 40)])
def test_no_allocation_forms(engine, nx, ny, gates):
    import torch
    from viennaemc_gb300 import _lib as L
    dev = _bar(nx, ny, gates)
    pot, conc = _start(dev, nx)
    sim = _sim(engine, dev, True)
    want, info = _solve(sim, pot, conc)
    sim.close()
    desc = dev.desc()
    d_pot, d_conc = (torch.tensor(v, device="cuda") for v in (pot, conc))
    rel, cyc = C.c_double(), C.c_int32()
    torch.cuda.synchronize()
    L.check(L.lib().emcg_poisson_solve_noalloc(
        C.byref(desc), C.c_void_p(d_pot.data_ptr()), C.c_void_p(d_conc.data_ptr()), 1, 0, 1e-10,
        200, None, C.byref(rel), C.byref(cyc)))
    assert abs(cyc.value - info[1]) <= 1 and rel.value <= 1e-10
    assert np.max(np.abs(d_pot.cpu().numpy() - want)) <= 1e-8


# (columns, rows): two row groups whose last rows are missing in some CTAs; the widest
# grid of two groups; four groups and an odd width; a column of two rows too many
@pytest.mark.parametrize("nx,ny", [(401, 197), (511, 120), (303, 229), (255, 301), (305, 263)])
def test_column_sweeps_equal_one_launch_per_phase(engine, nx, ny):
    dev = _bar(nx, ny, gates=3)
    pot, conc = _start(dev, nx + ny)
    sim = _sim(engine, dev, True)
    assert sim.poisson_mode(-1) > 1
    a, ia = _solve(sim, pot, conc)
    sim.poisson_mode(0)
    b, ib = _solve(sim, pot, conc)
    sim.close()
    assert ia[1] == ib[1]
    assert np.max(np.abs(a - b)) <= 1e-13 * max(1.0, np.abs(b).max())
