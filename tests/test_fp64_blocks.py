"""The double engines' building blocks against the plain expressions they stand for,
natively compiled and through the engines."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


def _native(tmp_path, name):
    exe = tmp_path / name
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    f"-I{ROOT}/viennaemc_gb300/csrc", f"{ROOT}/tests/native/{name}.cpp", "-o",
                    str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


def test_comparisons_fixed_point_and_steps(tmp_path):
    """The steps round once at the result's size (half a unit); what they leave out is
    5 e^3 / 16 with |e| < 2^-19 (0.02 units) and r^3 with r < 2^-20 (0.01)."""
    below, fixed, rsqrt, rcp = _native(tmp_path, "fp64_check")
    assert (below, fixed) == ("0", "0")
    assert float(rsqrt) <= 0.53 and float(rcp) <= 0.52


@pytest.mark.gpu
def test_roots_and_quotients_on_the_gpu(engine, tmp_path):
    """The hardware's approximations cut their argument and their result to 20 fraction
    bits, so they are within 2^-19; from them the steps' bounds, and sqrtD and divD,
    corrected once at the result's size, half a unit and a hundredth; at the ends of
    their ranges the library's results or their neighbours, outside its own."""
    exe = tmp_path / "fp64_gpu_check"
    lib = engine._lib
    subprocess.run([lib._nvcc(), lib.ARCH, "-O3", "-std=c++17", f"-I{lib.INCLUDE}",
                    f"-I{lib.CSRC}", f"{ROOT}/tests/native/fp64_gpu_check.cu", "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    low, approx, rsqrt, rcp, root, quotient, edges = map(float, out)
    assert low == 0 and approx <= 2.0  # approx: in 2^-20
    assert rsqrt <= 0.53 and rcp <= 0.52 and root <= 0.51 and quotient <= 0.51
    assert edges == 0


def _bar(nx=41, ny=31, h=1e-9):
    from viennaemc_gb300 import device as D
    from viennaemc_gb300.physics import silicon_material
    lx, ly = (nx - 1) * h, (ny - 1) * h
    dev = D.Device(silicon_material(), (lx, ly), (h, h))
    dev.addConstantDopingRegion((0, 0), (lx, ly), 1e24)
    dev.addOhmicContact(D.XMIN, 0.0, (0,), (ly,))
    dev.addOhmicContact(D.XMAX, 0.0, (0,), (ly,))
    return dev


def _resting(engine, pos):
    """Electrons at rest at pos (n x 2) without an event ahead; k of -0, so that a
    field-free flight leaves a coordinate of -0 as it is."""
    n = len(pos)
    z = np.zeros(n)
    return engine.ParticleState.from_arrays(
        kx=-z, ky=-z, kz=-z, px=pos[:, 0], py=pos[:, 1], pz=z, energy=z,
        tau=np.full(n, 1.0), grain_tau=np.full(n, 1.0), valley=np.zeros(n, np.int32),
        sub=np.zeros(n, np.int32), region=np.zeros(n, np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_minus_zero_is_inside_the_device(engine, precision):
    """Removal at a contact is for positions < 0 or > max (include/emcParticleDrift.hpp:
    41-66): -0 and max itself stay."""
    from viennaemc_gb300 import device as D
    dev = _bar()
    pt = engine.physics.silicon_electron("refbulk", n_levels=100, max_energy=4.0)
    sim = D.DeviceSimulation(dev, pt, scheme=D.NGP, capacity=64, dt=1e-16, precision=precision)
    y = dev.max_pos[1] / 2
    pos = np.array([[-0.0, y], [0.0, y], [dev.max_pos[0], y], [-1e-12, y], [3e-9, y]])
    sim.set_state(_resting(engine, pos))
    netto = sim.move(step=0)
    st = sim.get_state()
    sim.close()
    assert netto.sum() == 1 and st.n == 4  # the one outside
    assert sorted(st.px) == sorted(np.float32(pos[[0, 1, 2, 4], 0]) if precision == "fp32"
                                   else pos[[0, 1, 2, 4], 0])


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1e-9, 0.5e-9, 0.7e-9])
@pytest.mark.parametrize("scheme", ["ngp", "cic"])
def test_grid_lookups_beside_whole_and_half_numbers(engine, scheme, h):
    """The node of a position (the nearest, and the lower one with its weight) is that of
    v / h, also a few units in the last place from k h and (k + 1/2) h, and between."""
    from viennaemc_gb300 import _lib as L
    from viennaemc_gb300 import device as D
    nx, ny = 201, 31
    dev = _bar(nx, ny, h)
    pt = engine.physics.silicon_electron("refbulk", n_levels=100, max_energy=4.0)
    rs = np.random.default_rng(17)
    k = rs.integers(0, 2 * (nx - 1), 6000)
    x = np.abs(k * (h / 2) * (1 + rs.integers(-4, 5, k.size) * 2.0 ** -53))
    x[4000:] = rs.random(2000) * (nx - 1) * h
    x[5000:] = (k[5000:] * (h / 2)) * (1 + (rs.random(1000) - 0.5) * 2.0 ** -17)
    x = np.clip(x, 0.0, dev.max_pos[0])
    y = np.full(x.size, 3 * h)
    sim = D.DeviceSimulation(dev, pt, scheme=D.NGP if scheme == "ngp" else D.CIC,
                             capacity=x.size)
    sim.set_state(_resting(engine, np.stack([x, y], 1)))
    sim.assign()
    got = sim.get_grid(L.GRID_NRPART).reshape(ny, nx) / sim.carriers
    sim.close()
    want = np.zeros((ny, nx))
    if scheme == "ngp":
        q = x / h
        near = np.floor(q) + (q - np.floor(q) >= 0.5)
        np.add.at(want, (np.full(x.size, int(np.rint(y[0] / h))), near.astype(int)), 1.0)
        assert np.array_equal(got, want)
    else:
        m, w = [], []
        for v in (x, y):
            q = v / h
            m.append(np.floor(q).astype(int))
            w.append(q - np.floor(q))
        for dx in (0, 1):
            for dy in (0, 1):
                cx, cy = m[0] + dx, m[1] + dy
                on = (cx < nx) & (cy < ny)
                wt = (w[0] if dx == 0 else 1 - w[0]) * (w[1] if dy == 0 else 1 - w[1])
                np.add.at(want, (cy[on], cx[on]), wt[on])
        # a weight is off by a unit in the last place of q < 256 at most
        assert np.max(np.abs(got - want)) <= 2.0 ** -45 * np.max(np.bincount(m[0]) * 2 + 2)
