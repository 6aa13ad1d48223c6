"""Which form the Poisson solves of test_gpu_poisson_large.py take: the comparisons
there hold for any, so a plan that finds no cluster would pass them unseen."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_poisson_large import _bar, _sim, _solve, _start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,fp32", [(601, 301, True), (1203, 137, True), (399, 398, False),
                                        (801, 401, True)])
def test_large_grids_have_a_tail_in_a_cluster(engine, nx, ny, fp32):
    sim = _sim(engine, _bar(nx, ny), fp32)
    ctas, level, tail = sim.poisson_form()
    assert ctas == 0 and level >= 1 and tail > 1
    sim.poisson_mode(0)
    assert sim.poisson_form() == (0, 0, 0)
    sim.poisson_mode(1)
    assert sim.poisson_form() == (0, level, tail)
    # a bound holds for the tail too
    sim.set_poisson_cluster(8)
    assert sim.poisson_form()[0] == 0 and 0 < sim.poisson_form()[2] <= 8
    sim.close()


@pytest.mark.parametrize("nx,ny", [(41, 31), (201, 101), (401, 201), (511, 120)])
def test_grids_that_fit_are_one_cluster(engine, nx, ny):
    sim = _sim(engine, _bar(nx, ny), True)
    assert sim.poisson_form() == (sim.poisson_mode(-1), 0, 0) and sim.poisson_form()[0] >= 1
    sim.close()


# one cluster; a tail; more coefficient tuples than the class table's 64 (one for each
# gate's coupling and some for the grid's edges)
@pytest.mark.parametrize("nx,ny,gates,form", [(201, 101, 0, "cluster"), (360, 361, 0, "tail"),
                                              (301, 61, 40, "cluster"), (301, 61, 61, "phases")])
def test_no_allocation_solve_takes_its_form(engine, nx, ny, gates, form):
    """... and gives the allocating solve's potential (1e-8, as test_zz_no_alloc)."""
    import torch
    L = engine._lib
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
    out = [C.c_int32() for _ in range(3)]
    L.check(L.lib().emcg_poisson_noalloc_form(*map(C.byref, out)))
    ctas, level, tail = (v.value for v in out)
    assert (ctas > 0, level > 0, tail > 0) == {"cluster": (True, False, False),
                                               "tail": (False, True, True),
                                               "phases": (False, False, False)}[form]
    assert abs(cyc.value - info[1]) <= 1 and rel.value <= 1e-10
    assert np.max(np.abs(d_pot.cpu().numpy() - want)) <= 1e-8
