"""The device sort and scan at the edges of their tiles (2048 pairs a tile, a
warp's 256; 8192 values a scan tile) and past the tile count up to which a
scatter block sums the earlier tiles itself: particles at rest re-bin into
exactly the host's stable order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 255, 257, 2047, 2048, 2049, 8191, 8193, 20000, 330001, 700001])
@pytest.mark.parametrize("spread", [3.0, 400.0, 3.0e7])
def test_rebin_of_particles_at_rest(n, spread):
    from sharc.volrus_b200 import PARTICLE, PointDataGrid, advect_particles_euler, make_uniform_velocity
    rng = np.random.default_rng([n, int(spread)])
    parts = np.zeros(n, PARTICLE)
    parts["position"] = rng.uniform(-spread, spread, (n, 3))
    parts["id"] = np.arange(n)
    pg, host = PointDataGrid(1.0), PointDataGrid(1.0)
    pg.particles = parts.copy()
    host.insert_batch(parts)
    advect_particles_euler(pg, make_uniform_velocity(1.0, (0.0, 0.0, 0.0)), 1.0)
    assert np.array_equal(pg.particles["id"], host.particles["id"])
    assert np.array_equal(pg.particles["position"], host.particles["position"])
    assert np.array_equal(pg.leaf_origins, host.leaf_origins)
    assert np.array_equal(pg.leaf_start, host.leaf_start)
