"""The Coulomb sums at the edges of their tiles, groups and target blocks, and
pairs whose float r^2 is subnormal or zero (the packed float term hands those
tiles to the plain one).  Tolerances as in test_p2p.py: the double sums differ
from the oracle's by the order of the additions, the float ones by the
rounding of the nearest pairs' positions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
Q = 1.60219e-19


def _rel(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


@pytest.mark.parametrize("n,images", [(1, 0), (1, 1), (2, 0), (7, 0), (9, 1), (127, 0), (129, 0),
                                      (255, 0), (256, 0), (257, 0), (511, 1), (513, 0), (1025, 0),
                                      (2431, 0)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-4)])
@pytest.mark.parametrize("cut", [1e9, 0.0])
def test_sums_at_tile_edges(engine, oracle, n, images, precision, tol, cut):
    from viennaemc_gb300 import p2p
    rs = np.random.default_rng(100 + n)
    box = 1e-7
    pos = rs.random((3, n)) * box
    q = np.where(rs.random(n) < 0.5, -Q, 1.5 * Q)
    f, p = p2p.coulomb(pos, q, cut, box, images, precision)
    fo, po = oracle.p2p_coulomb(pos, q, cut, box, images)
    # against the size of the terms: a charge's own periodic copies cancel
    term = Q * Q / box ** 2
    assert np.max(np.abs(f - fo)) <= tol * max(np.max(np.abs(fo)), term)
    assert _rel(p, po) <= tol


@pytest.mark.parametrize("at", [0, 200, 300])
def test_float_pairs_below_the_smallest_normal(engine, at):
    """Two charges 8e-20 m apart (r^2 subnormal in float) among 600 others, and
    two that coincide: the others' sums, the close pair's force at the cutoff and
    every potential are those of the double engine; the coinciding pair's force
    has no direction in either."""
    from viennaemc_gb300 import p2p
    rs = np.random.default_rng(5)
    n = 602
    pos = rs.random((3, n)) * 1e-7
    q = np.where(np.arange(n) % 2 == 0, -Q, Q)
    pos[:, at] = 0.0
    pos[:, at + 1] = (8e-20, 0.0, 0.0)
    f, p = p2p.coulomb(pos, q, 1e9, precision="fp32")
    g, r = p2p.coulomb(pos, q, 1e9, precision="fp64")
    assert np.all(np.isfinite(f)) and _rel(f, g) <= 1e-4 and _rel(p, r) <= 1e-4
    pos[:, at + 1] = 0.0
    f, p = p2p.coulomb(pos, q, 1e9, precision="fp32")
    g, r = p2p.coulomb(pos, q, 1e9, precision="fp64")
    ok = np.ones(n, bool)
    ok[[at, at + 1]] = False
    assert _rel(f[:, ok], g[:, ok]) <= 1e-4 and _rel(p, r) <= 1e-4
    assert np.all(np.isnan(f[:, ~ok])) and np.all(np.isnan(g[:, ~ok]))
