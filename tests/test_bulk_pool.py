"""The double engine's pooled step kernel (mode 0) against the block-queued one
(mode 1), which runs the plain per-particle step: the same Philox counters, so
the same trajectories bar last-ulp branch flips.  And its integer forms of the
uniform draw and the table level, and its log, against the expressions they
stand for (host, compiled natively)."""
import os
import subprocess

import numpy as np
import pytest

from test_host import L_FRAMES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _native(tmp_path, name):
    exe = tmp_path / name
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    f"-I{ROOT}/viennaemc_gb300/csrc", f"{ROOT}/tests/native/{name}.cpp", "-o",
                    str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


def test_log_of_the_draws(tmp_path):
    """Within 1.01 units in the last place of the extended-precision log (the
    table sum and the last addition round once each at most half a unit)."""
    worst, rms, _, specials = _native(tmp_path, "log_check")
    assert float(worst) <= 1.01 and float(rms) < 0.29 and specials == "1"


def test_integer_draw_and_level(tmp_path):
    assert _native(tmp_path, "draws_check") == ["0"]


def _tilted(engine):
    """Two valleys, the upper one with eight subvalleys whose axes are not the
    device's."""
    from viennaemc_gb300 import physics as P
    mat = P.silicon_material()
    pt = P.Electron(1000, 2.0)
    P.add_x_valley(pt, 0.19)
    v = P.NonParabolicAnisotropValley([0.8, 0.2, 0.2], pt.getMass(), 8, 0.3, 0.15)
    for s, f in enumerate(L_FRAMES):
        v.setSubValleyEllipseCoordSystem(s, *f)
    pt.addValley(v)
    for k in (0, 1):
        pt.addScatterMechanism([0], P.AcousticScatterMechanism(k, 9.0, 300.0, mat.rho,
                                                               mat.velSound))
    up, down = {s: [0, 3, 5] for s in range(3)}, {s: [s % 3] for s in range(8)}
    for cls in (P.ZeroOrderInterValleyAbsorptionScatterMechanism,
                P.ZeroOrderInterValleyEmissionScatterMechanism):
        pt.addScatterMechanism([0], cls("XL", 0, up, 2e10, 0.03, 300.0, mat.rho, 1))
        pt.addScatterMechanism([0], cls("LX", 1, down, 2e10, 0.03, 300.0, mat.rho, 0))
    pt.initScatterTables()
    return pt


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["silicon", "grain", "tilted"])
@pytest.mark.parametrize("counts", [(1,), (31, 0, 33), (600, 29300), (60013,), (120001,)])
def test_pooled_kernel_equals_queued_kernel(engine, model, counts):
    """Pools of one electron, of a partial warp, of 16 to 32, 33 to 64 and 65 to
    96 electrons, several ensembles and more than one wave; both step launches
    of 9 steps, so the window and the sums' tail are passed.  A trajectory may
    branch on a last-ulp difference, as between the other kernels."""
    pt = _tilted(engine) if model == "tilted" else \
        engine.physics.silicon_electron("jacoboni", grain=(0.3, 2e13) if model == "grain" else None)
    specs = [engine.EnsembleSpec(0, n, 2e6, (1, 2, 3), (2e-7, 3e-7, 1e-6), 1e-15, 21 + e, e)
             for e, n in enumerate(counts)]
    runs = []
    for mode in (0, 1):
        b = engine.BulkBatch([pt], specs, "fp64")
        b.set_launch(queued=mode, steps_per_launch=9)
        for e in range(len(counts)):
            b.init_particles(e)
        obs = b.step(22)
        runs.append(([b.get_state(e) for e in range(len(counts))], obs))
        b.close()
    for e, n in enumerate(counts):
        a, q = runs[0][0][e], runs[1][0][e]
        # with grains the two kernels draw them from other Philox calls: only the
        # electrons without a grain event agree (a step has one for 2 in 100)
        same = np.ones(n, bool) if model != "grain" else np.abs(a.grain_tau - q.grain_tau) < 1e-20
        bad = (a.valley != q.valley) | (a.sub != q.sub)
        for f in ("kx", "ky", "kz", "px", "py", "pz", "energy", "tau"):
            x, y = getattr(a, f), getattr(q, f)
            bad |= np.abs(x - y) > 1e-12 * np.max(np.abs(y), initial=0.0)
        assert n == 0 or same.mean() > 0.5 or n < 10
        assert (bad & same).sum() <= n // 1000, (e, (bad & same).sum())
        oa, oq = runs[0][1][e], runs[1][1][e]
        assert np.array_equal(oa[:, :, 2].sum(axis=1), np.full(22, n))
        if model != "grain" and n:
            assert np.allclose(oa[:, :, 2], oq[:, :, 2], atol=2)
            assert np.allclose(oa.sum(axis=1)[:, 0], oq.sum(axis=1)[:, 0], rtol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("block", [0, 64])
def test_autotune_of_a_double_engine(engine, block):
    """The pooled kernel has one shape: it is tried once beside the three block-queued
    ones, and where it wins (it does, threefold) the block size and the register cap
    of the other steps stay as they were, automatic ones too."""
    spec = engine.EnsembleSpec(0, 20000, 1e6, (1, 0, 0), (1e-6,) * 3, 1e-15, 3)
    b = engine.BulkBatch([engine.silicon_electron("jacoboni")], [spec], "fp64")
    b.set_launch(block_threads=block, steps_per_launch=7, min_blocks=3)
    b.init_particles(0)
    b.step(2)
    before = b.launch()
    cfg = b.autotune(5)
    assert cfg["steps_used"] == 2 * 4 * 5 and cfg["queued"] == 0
    assert cfg["block_threads"] == before["block_threads"] == (block or 256)
    assert cfg["min_blocks"] == 3 and b.launch() == before
    assert np.array_equal(b.step(3)[0, :, :, 2].sum(axis=1), np.full(3, 20000))
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [20, 20000])
def test_event_limit_of_a_step(engine, n):
    """An electron may have 65,536 events in a step, real or self-scattering: a step of
    62,000 mean free flights (249 is a standard deviation) runs, one of 69,000 does not,
    in the pooled kernel as in the block-queued one.  Without a field the first gives
    equal electrons, bar last-ulp branch flips."""
    pt = engine.silicon_electron("jacoboni")
    got = {}
    for flights in (62000, 69000):
        for mode in (0, 1):
            spec = engine.EnsembleSpec(0, 20, 0.0, (1, 0, 0), (1e-6,) * 3, 1e-15, 3)
            more = [engine.EnsembleSpec(0, n - 20, 0.0, (1, 0, 0), (1e-6,) * 3, 1e-18, 4)] * (n > 20)
            b = engine.BulkBatch([pt], [spec] + more, "fp64")
            tau = float(np.atleast_1d(b.get_rates(0)[1])[0])
            b.close()
            spec = engine.EnsembleSpec(0, 20, 0.0, (1, 0, 0), (1e-6,) * 3, flights * tau, 3)
            b = engine.BulkBatch([pt], [spec] + more, "fp64")
            b.set_launch(queued=mode)
            for e in range(1 + len(more)):
                b.init_particles(e)
            if flights == 69000:
                with pytest.raises(engine._lib.EmcgError, match="gave up"):
                    b.step(1)
            else:
                b.step(1)
                got[mode] = b.get_state(0)
            b.close()
    a, q = got[0], got[1]
    bad = (a.valley != q.valley) | (a.sub != q.sub)
    for f in ("kx", "ky", "kz", "energy", "tau"):
        x, y = getattr(a, f), getattr(q, f)
        bad |= np.abs(x - y) > 1e-9 * np.max(np.abs(y))
    assert bad.sum() <= 1


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["silicon", "tilted"])
@pytest.mark.parametrize("n", [7, 600, 60013, 120001])
@pytest.mark.parametrize("box,dt,spread", [((1e-6, 1e-6, 1e-6), 1e-15, 4.0),
                                           ((1e-8, 3e-8, 2e-9), 2e-14, 1.0),
                                           ((2e-9, 2e-9, 5e-9), 3e-15, 2.5)])
def test_periodic_box_as_the_reference_wraps_it(engine, model, n, box, dt, spread):
    """One box length is added or taken after a flight (basicBulkParticleHandler.hpp:
    600-613): electrons that start outside the box come nearer by one a flight, and
    flights longer than it end outside.  Against the block-queued kernel, which wraps
    each flight; positions within 1e-9 of a box."""
    pt = _tilted(engine) if model == "tilted" else engine.physics.silicon_electron("jacoboni")
    spec = engine.EnsembleSpec(0, n, 2e6, (1, 2, 3), box, dt, 21)
    rs = np.random.default_rng(n)
    start = (rs.random((3, n)) - 0.5) * 2 * spread + 0.5
    got = []
    for mode in (0, 1):
        b = engine.BulkBatch([pt], [spec], "fp64")
        b.set_launch(queued=mode)
        b.init_particles(0)
        st = b.get_state(0)
        for f, x, L in zip(("px", "py", "pz"), start, box):
            getattr(st, f)[:] = x * L
        st.tau[::5] *= -1.0  # a timer that ran out before the call
        b.set_state(0, st)
        b.step(3)
        got.append(b.get_state(0))
        b.close()
    a, q = got
    bad = (a.valley != q.valley) | (a.sub != q.sub)
    for f, L in zip(("px", "py", "pz"), box):
        bad |= np.abs(getattr(a, f) - getattr(q, f)) > 1e-9 * L
    assert bad.sum() <= n // 1000
