"""The double engine's move with its events queued per block: every electron,
some, or none with an event inside the step, in blocks that are full and not,
against the oracle on the same Philox stream (1e-12, as test_gpu_device.py)."""
import numpy as np
import pytest

from conftest import golden
from test_gpu_device import (DEVICE_CASES, FIELDS_F, ENG, RTOL, _engine_state, _oracle_device,
                             _oracle_model, _sim, flavour)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", DEVICE_CASES)
@pytest.mark.parametrize("n,share", [(1, 1.0), (33, 1.0), (256, 1.0), (257, 0.5), (700, 1.0),
                                     (700, 0.0)])
def test_queued_move_matches_oracle(engine, oracle, case, n, share):
    from viennaemc_gb300 import _lib as L
    g = golden(case)
    n = min(n, len(g["s0_E"]))
    sim, dev, pt = _sim(engine, g, case, seed=0xABBA)
    odev = _oracle_device(oracle, g)
    m, _ = _oracle_model(oracle, g)
    scheme, _, _ = flavour(g)
    dt = float(g["params"][1])
    d = {f: g[f"s0_{f}"][:n].copy() for f in oracle.STATE_F + oracle.STATE_I}
    rs = np.random.default_rng(n)
    # an event inside the step for a share of the electrons, none for the others
    d["tau"] = np.where(rs.random(n) < share, dt * (0.02 + 0.96 * rs.random(n)),
                        dt * (1.5 + rs.random(n)))
    cur = oracle.State.from_dict(d)
    est = engine.ParticleState.from_arrays(
        pz=np.zeros(n), **{ENG.get(f, f): d[f] for f in FIELDS_F},
        **{f: d[f] for f in ("valley", "sub", "region")})
    sim.set_state(est)
    sim.set_grid(L.GRID_POTENTIAL, g["pot1"])
    sim.efield()
    Ex, Ey = odev.efield(g["pot1"], scheme)
    netto = sim.move(step=5)
    rc, onet, _ = odev.move(m, scheme, cur, Ex, Ey, dt, oracle.RngState(oracle.RNG_PHILOX, 0xABBA, 0),
                            5)
    assert np.array_equal(netto, onet)
    st = sim.get_state()
    assert st.n == cur.n
    for f in FIELDS_F:
        a, b = getattr(st, ENG.get(f, f)), getattr(cur, f)[:cur.n]
        assert np.max(np.abs(a - b), initial=0.0) <= RTOL * max(np.abs(b).max(initial=0.0), 1e-300)
    for f in ("valley", "sub", "region"):
        assert np.array_equal(getattr(st, f), getattr(cur, f)[:cur.n])
    sim.close()
