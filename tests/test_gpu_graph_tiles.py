"""Graph replay beside steps that work on another tile list.  The double engine's
pooled launches and its Coulomb steps (thread blocks) share one tile buffer: 32-thread
blocks need a longer list than the pools, so the buffer moves between two replays."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [30000, 40007])
def test_replay_after_the_tile_buffer_moved(engine, n):
    spec = engine.EnsembleSpec(0, n, 1e6, (1, 2, 3), (1e-6,) * 3, 1e-15, 5, 0)
    runs = []
    for graph in (True, False):
        b = engine.BulkBatch([engine.silicon_electron("jacoboni")], [spec], "fp64")
        b.set_launch(block_threads=32)
        b.set_graph(graph)
        b.init_particles(0)
        obs = [b.step(3)]
        b.set_coulomb(11.7)
        obs.append(b.step(1))
        b.set_coulomb(11.7, enable=False)
        obs += [b.step(3), b.step(3)]
        runs.append((b.get_state(0), np.concatenate(obs, axis=1)))
        b.close()
    (a, oa), (q, oq) = runs
    # the same kernels on the same electrons: equal; the sums' atomics add some 1300
    # values in another order, velocities of both signs up to 1e6 m/s
    for f in ("kx", "ky", "kz", "px", "py", "pz", "energy", "tau", "valley", "sub"):
        assert np.array_equal(getattr(a, f), getattr(q, f)), f
    assert np.allclose(oa[..., 0], oq[..., 0], rtol=1e-10, atol=0)
    assert np.allclose(oa[..., 1], oq[..., 1], rtol=0, atol=1e-12 * n * 1e6)
    assert np.array_equal(oa[0, :, :, 2].sum(axis=1), np.full(10, n))
