"""Particles in, beside and far from the leaves of their velocity grids, mixed
within warps in every proportion, against the oracle bit for bit; and active
counts of grids around the number of leaves that are counted on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(seed, leaves, voxel_size=1.0):
    from sharc.volrus_b200.grid import Grid, VoxelTransform
    g = np.random.default_rng(seed)
    c = np.stack(np.unravel_index(g.permutation(6 ** 3)[:leaves], (6,) * 3), 1) - 3
    m = np.packbits(g.random((leaves, 512)) < 0.7, axis=1, bitorder="little").view(np.uint64)
    return Grid.from_arrays((c * 8).astype(np.int32), m, g.uniform(-1, 1, (leaves, 512)).astype(np.float32), 0.25,
                            VoxelTransform.uniform(voxel_size))


@pytest.mark.parametrize("leaves", [1, 100, 216])
@pytest.mark.parametrize("span", [20.0, 24.0, 30.0, 500.0])
@pytest.mark.parametrize("shared", [True, False])
def test_positions_match_the_oracle(oracle, leaves, span, shared):
    from sharc.volrus_b200.tools import VelocityField, advect_particles, advect_particles_euler
    gs = [_grid(a, leaves if a == 0 else min(leaves + 7 * a, 216), 1.0 if shared else 1.0 + 0.25 * a) for a in range(3)]
    vel = VelocityField(*gs)
    og = [oracle.OGrid.from_arrays(*g.to_arrays(), g.background, g.transform.voxel_size) for g in gs]
    for n in (1, 31, 33, 1000):
        p = np.random.default_rng(n).uniform(-span, span, (n, 3))
        for rk4, f in ((True, advect_particles), (False, advect_particles_euler)):
            for dt in (0.5, 20.0):
                assert np.array_equal(f(p, vel, dt), oracle.advect_particles(*og, p, dt, rk4=rk4)), (n, rk4, dt)


@pytest.mark.parametrize("leaves", [1, 31, 32, 33, 200])
def test_active_count(leaves):
    from sharc.volrus_b200.tools import DeviceGrid
    g = _grid(9, leaves)
    want = int(np.unpackbits(g.to_arrays()[1].view(np.uint8)).sum())
    d = DeviceGrid.upload(g)
    assert d.info()[:2] == (leaves, want)
    d.close()
