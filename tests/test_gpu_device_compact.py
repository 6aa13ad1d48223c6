"""The device step's fused kernels (the compaction and the injection assign the
charge) against the same stages called one by one, for every particle-mesh scheme,
with so few blocks that each one sums the counts before it and with so many (more
than 4096 blocks of 1024 particles) that they are scanned first."""
import numpy as np
import pytest

from conftest import golden
from test_gpu_device import DEVICE_CASES, _electron, _host_device, flavour, surfaces

pytestmark = pytest.mark.gpu

FEW, MANY = 1 << 15, 4096 * 1024 + 1


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("capacity", [FEW, MANY])
@pytest.mark.parametrize("scheme", ["ngp", "cic", "nec"])
def test_fused_step_equals_its_stages(engine, scheme, capacity, precision):
    from viennaemc_gb300 import _lib as L
    from viennaemc_gb300 import device as D
    case = DEVICE_CASES[0]
    g = golden(case)
    _, pot_init, vwd = flavour(g)

    def sim():
        dev = _host_device(g, pot_init)
        s = D.DeviceSimulation(dev, _electron(engine, dev, None, surfaces(g)),
                               scheme=getattr(L, "PM_" + scheme.upper()), dt=float(g["params"][1]),
                               seed=11, capacity=capacity, precision=precision,
                               potential_init=pot_init, round_counts=vwd,
                               tau_region_is_valley=vwd)
        s.calcEquilibriumCharacteristics()
        return s

    a, b = sim(), sim()
    steps, s0, rows = 4, b.step_index, []
    net = a.performEMCStep(steps)
    for s in range(steps):
        b.poisson(equilibrium=False, reset_bc=(s == 0))
        b.efield()
        moved = b.move(step=s0 + s)
        rows.append(moved - b.contacts(step=s0 + s))
        b.assign()
    assert np.array_equal(net, np.array(rows))
    for grid in (L.GRID_POTENTIAL, L.GRID_NRPART, L.GRID_CONC):
        assert np.array_equal(a.get_grid(grid), b.get_grid(grid)), grid
    sa, sb = a.get_state(), b.get_state()
    assert sa.n == sb.n == a.num_particles()
    for f in ("kx", "ky", "kz", "energy", "px", "py", "tau", "valley", "sub", "region"):
        assert np.array_equal(getattr(sa, f), getattr(sb, f)), f
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx", [5, 512, 513])
def test_injection_fills_every_reservoir_node(engine, nx, precision):
    """Up to 1024 reservoir nodes every block of the injection forms the nodes' numbers
    itself, beyond one block does so first: after a step each contact node holds its
    expected number of carriers, rounded up (nearest-node charge)."""
    from viennaemc_gb300 import _lib as L
    from viennaemc_gb300 import device as D
    from viennaemc_gb300.physics import silicon_material
    h, ny = 1e-9, 6
    dev = D.Device(silicon_material(), ((nx - 1) * h, (ny - 1) * h), (h, h))
    dev.setDeviceWidth(6.7e-7)  # 6.7 electrons a cell, 3.35 at a contact node
    dev.addConstantDopingRegion((0, 0), ((nx - 1) * h, (ny - 1) * h), 1e25)
    dev.addOhmicContact(D.YMIN, 0.0, (0,), ((nx - 1) * h,))
    dev.addOhmicContact(D.YMAX, 0.05, (0,), ((nx - 1) * h,))
    pt = engine.physics.silicon_electron("refbulk", n_levels=500, max_energy=4.0)
    sim = D.DeviceSimulation(dev, pt, scheme=D.NGP, dt=1e-16, seed=9, precision=precision)
    sim.calcEquilibriumCharacteristics()
    n0 = sim.num_particles()
    netto = sim.performEMCStep(3)
    assert sim.num_particles() == n0 - int(netto.sum())
    held = sim.get_grid(L.GRID_NRPART).reshape(ny, nx)
    assert np.all(held[[0, -1], 1:-1] == 4.0)
    sim.close()
