"""The bit-mask forms of the crate's band tools where masks could go wrong:
values whose products underflow, infinities, NaN, signed zeros and denormals,
leaves far apart, and half-empty neighbourhoods; bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1e-40, -1e-40, 1e-30, -1e-30, 3e-23, -3e-23, 2.0 ** -62, -2.0 ** -62, 2.0 ** -63, 0.5,
                    -0.5, 3e38, -3e38, np.inf, -np.inf, np.nan], np.float32)


def special_grid(seed, n, spread, fill, mix):
    """Random leaves; `mix` of the values are drawn from SPECIAL, the rest normal."""
    from sharc.volrus_b200 import Grid
    rng = np.random.default_rng(seed)
    o = np.unique(rng.integers(-spread, spread, (n, 3)), axis=0).astype(np.int32) * 8
    n = len(o)
    on = rng.random((n, 512)) < fill
    v = np.where(rng.random((n, 512)) < mix, rng.choice(SPECIAL, (n, 512)), rng.normal(0, 1, (n, 512)))
    m = np.packbits(on, axis=1, bitorder="little").view(np.uint64)
    return Grid.from_arrays(o, m, v.astype(np.float32), 2.0, None)


def to_oracle(oracle, g):
    o, m, v = g.to_arrays()
    return oracle.OGrid.from_arrays(o, m, v, g.background, g.transform.voxel_size, g.transform.origin, g.affine.mat,
                                    g.affine.voxel_size)


@pytest.mark.parametrize("seed,n,spread,fill,mix", [(1, 40, 2, 0.7, 0.0), (2, 40, 2, 0.7, 0.4), (3, 60, 3, 0.5, 1.0),
                                                    (4, 1, 1, 0.9, 0.3), (5, 300, 100000, 0.2, 0.1),
                                                    (6, 33, 40, 1.0, 0.05)])
def test_crossings_match_oracle(oracle, seed, n, spread, fill, mix):
    from sharc.volrus_b200 import find_zero_crossings
    g = special_grid(seed, n, spread, fill, mix)
    assert np.array_equal(find_zero_crossings(g), to_oracle(oracle, g).zero_crossings())


@pytest.mark.parametrize("hw", [0.4, 1.0, 1.7, 2.0, 2.6, 3.0, 3.2, 4.0])
@pytest.mark.parametrize("seed,n,spread,fill,mix", [(7, 40, 2, 0.7, 0.02), (8, 25, 2, 1.0, 0.3), (9, 5, 50, 0.1, 0.0)])
def test_rebuild_rows_match_oracle(oracle, hw, seed, n, spread, fill, mix):
    """Windows of half size 0 to 3: whole rows up to 2, voxel windows above; sparse and crowded crossings."""
    from sharc.volrus_b200 import rebuild_narrow_band
    g = special_grid(seed, n, spread, fill, mix)
    og = to_oracle(oracle, g)
    rebuild_narrow_band(g, hw)
    og.rebuild(hw, brute=True)
    o1, m1, v1 = g.to_arrays()
    o2, m2, v2 = og.arrays()
    assert np.array_equal(o1, o2) and np.array_equal(m1, m2)
    assert np.array_equal(v1.view(np.uint32), v2.view(np.uint32))


@pytest.mark.parametrize("same", [True, False], ids=["one-transform", "own-transforms"])
@pytest.mark.parametrize("dt", [0.0, 0.37, 30.0])
@pytest.mark.parametrize("seed,n,fill", [(11, 1, 1.0), (12, 3, 0.01), (13, 120, 0.3), (14, 40, 0.9)])
def test_advect_sampled_fields_match_oracle(oracle, same, dt, seed, n, fill):
    """Velocity grids over part of the level set's leaves, with one transform or three; samples inside the hinted
    neighbourhood, across its faces and far outside it; leaves without active voxels."""
    from sharc.volrus_b200 import VelocityField, VoxelTransform, advect_level_set
    g = special_grid(seed, n, 2, fill, 0.02)
    g._m[::5] = 0
    comps = []
    for a in range(3):
        v = special_grid(seed + 20 + a, n, 2, 0.8, 0.0)
        if not same:
            v.set_transform(VoxelTransform.uniform((1.0, 0.75, 1.5)[a]))
        comps.append(v)
    out = advect_level_set(g, VelocityField(*comps), dt)
    og = to_oracle(oracle, g).advect(*[to_oracle(oracle, c) for c in comps], dt)
    o1, m1, v1 = out.to_arrays()
    o2, m2, v2 = og.arrays()
    assert np.array_equal(o1, o2) and np.array_equal(m1, m2)
    assert np.array_equal(np.isnan(v1), np.isnan(v2))
    keep = ~np.isnan(v1)
    assert np.array_equal(v1.view(np.uint32)[keep], v2.view(np.uint32)[keep])


@pytest.mark.parametrize("iso", [0.0, 0.25])
@pytest.mark.parametrize("seed,n,spread,fill,mix", [(31, 30, 2, 1.0, 0.0), (32, 30, 2, 1.0, 0.3), (33, 1, 1, 1.0, 0.0),
                                                    (34, 40, 100000, 0.5, 0.0), (35, 200, 12, 0.3, 0.02)])
def test_mesh_tile_lists_match_oracle(oracle, iso, seed, n, spread, fill, mix):
    """Tiles from a bit per tile of the leaves' box, and from the sort where leaves lie far apart; crowded and empty
    tiles, infinities and NaN."""
    import ctypes as C
    from sharc.volrus_b200 import DeviceGrid, volume_to_mesh
    g = special_grid(seed, n, spread, fill, mix)
    m = volume_to_mesh(g, iso)
    v2, t2 = to_oracle(oracle, g).volume_to_mesh(iso)
    assert np.array_equal(m.triangles, t2)
    assert np.array_equal(np.isnan(m.vertices), np.isnan(v2))
    ok = ~np.isnan(v2)
    assert np.array_equal(m.vertices.view(np.uint64)[ok], v2.view(np.uint64)[ok])
    # the one-call form: counts, then as much as fits
    d = DeviceGrid.upload(g)
    nv, nt = C.c_size_t(), C.c_size_t()
    k = max(len(t2) // 2, 1)
    t = np.zeros((k, 3), np.uint32)
    d.ctx.check(d.ctx.lib.vlr_volume_to_mesh(d.ctx.handle, d.handle, C.c_float(iso), None, 0,
                                             t.ctypes.data_as(C.POINTER(C.c_uint32)), k, C.byref(nv), C.byref(nt)))
    assert (nv.value, nt.value) == (len(v2), len(t2))
    assert np.array_equal(t[:len(t2)], t2[:k])


@pytest.mark.parametrize("same", [True, False], ids=["one-transform", "own-transforms"])
@pytest.mark.parametrize("rk4", [True, False])
def test_particles_hinted_samples_match_oracle(oracle, same, rk4):
    """Particles inside and outside the velocity grids' leaves, steps within and beyond a leaf, far positions."""
    from sharc.volrus_b200 import VelocityField, VoxelTransform, advect_particles, advect_particles_euler
    comps = []
    for a in range(3):
        v = special_grid(40 + a, 30, 2, 0.8, 0.0)
        v.set_transform(VoxelTransform.uniform(0.5 if same else (0.5, 0.375, 0.75)[a]))
        comps.append(v)
    rng = np.random.default_rng(4)
    p = np.concatenate([rng.uniform(-9, 9, (5000, 3)), rng.uniform(-1e6, 1e6, (50, 3)), [[1e12, -1e12, 3.0]]])
    og = [to_oracle(oracle, c) for c in comps]
    for dt in (0.1, 9.0):
        got = (advect_particles if rk4 else advect_particles_euler)(p, VelocityField(*comps), dt)
        want = oracle.advect_particles(*og, p, dt, rk4)
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
