"""The windowed lambda transpose adds a voxel's terms in one order whatever the
size of the band, so a small band (wide kernel) and a large one that holds the
same leaves (past two waves of warps: narrow kernel) give the same bits there,
at reaches of one and of more voxels and windows of every depth in z."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere_leaves(center, r, half_width=3.0):
    """Leaves of a sphere's band, sorted (x, y, z)."""
    c = np.asarray(center, np.float64)
    lo = np.floor((c - r - 8) / 8).astype(int)
    side = int(np.ceil((2 * r + 16) / 8)) + 1
    q = np.stack(np.unravel_index(np.arange(side ** 3), (side,) * 3), 1) + lo
    q = q[np.abs(np.linalg.norm(q * 8 + 3.5 - c, axis=1) - r) < 11]
    loc = np.stack(np.unravel_index(np.arange(512), (8, 8, 8)), 1)
    phi = np.concatenate([np.linalg.norm(p[:, None] * 8 + loc[None] - c, axis=2) - r
                          for p in np.array_split(q, 16)]).astype(np.float32)
    on = np.abs(phi) < half_width
    keep = on.any(1)
    return ((q[keep] * 8).astype(np.int32),
            np.ascontiguousarray(np.packbits(on[keep], axis=1, bitorder="little")).view(np.uint64),
            phi[keep].clip(-half_width, half_width))


def _both():
    """A small sphere, and the same sphere beside a large one, leaves sorted."""
    a = _sphere_leaves((20.3, 40.0, 45.6), 12.4)
    b = _sphere_leaves((128.2, 96.0, 97.3), 72.0)
    o, m, p = (np.concatenate(x) for x in zip(a, b))
    s = np.lexsort((o[:, 2], o[:, 1], o[:, 0]))
    return a, (np.ascontiguousarray(o[s]), np.ascontiguousarray(m[s]), np.ascontiguousarray(p[s]))


def _compare(small, whole):
    """Gradients of both bands from the same lambda per voxel, compared on the small one."""
    line = 2 * 148 * 4 * 8  # chunks of up to 32 voxels that the wide kernel takes
    assert small.n_band < 32 * line < whole.n_band
    keys = [np.ravel_multi_index(tuple((f.band() + 64).T), (512,) * 3) for f in (small, whole)]
    lam = [((k * 2654435761 % 1000003) / 500001.5 - 1.0).astype(np.float32) for k in keys]
    for f in (small, whole):
        f.set_gather(1)
        f.forward()
    g = [f.backward(v)[0] for f, v in zip((small, whole), lam)]
    at = np.argsort(keys[1])[np.searchsorted(np.sort(keys[1]), keys[0])]
    assert np.array_equal(keys[1][at], keys[0])
    assert np.array_equal(g[1][at].view(np.uint32), g[0].view(np.uint32))
    assert np.abs(g[0]).max() > 0


@pytest.mark.parametrize("speed", [0.9, 0.999999, 1.0, 1.9, 3.9, 5.9])
def test_staggered(speed):
    from sharc.volrus_b200.adjoint import AdvectionFunction
    V = (np.random.default_rng(11).uniform(-1, 1, (3, 28, 28, 28)) * speed).astype(np.float32)
    if speed in (0.999999, 1.0):
        # a whole voxel a step and the largest speed below it that has a reach of one: foot offsets at an edge
        V = np.where(np.random.default_rng(12).random((3, 7, 7, 7)) < 0.5, -1, 1).repeat(4, 1).repeat(4, 2).repeat(4, 3)
        V = np.ascontiguousarray(V * speed, np.float32)
    fns = [AdvectionFunction(*leaves, V, 8.0, 1.0, 1e12 if speed <= 1.0 else 50.0, 3, 2) for leaves in _both()]
    _compare(*fns)
    for f in fns:
        f.close()


def test_level_set():
    from sharc.volrus_b200.adjoint import AdvectionFunction
    from sharc.volrus_b200.method import LevelSet, curl_noise
    vel = curl_noise(0, 48.0, 1.99, 1)  # displacements up to 0.96 voxels
    vel["domain"] = ((-64, -64, -64), (320, 320, 320))
    sets = [LevelSet.from_leaves(*leaves, vel, 1.0, integrator=2) for leaves in _both()]
    fns = [AdvectionFunction.from_level_set(ls, 3, 2) for ls in sets]
    _compare(*fns)
    for f in fns + sets:
        f.close()
