"""The windowed transpose at a band past two waves of warps, where it keeps one
candidate row in flight (smaller bands, three: the chunk tests), against the
FP64 oracle: a sphere of about 390,000 band voxels in a field whose foot
offsets differ within most leaves.

Two steps of FP32 arithmetic on |phi| <= 3: phi_K is within 2 * 8 * 3 * 2^-24 =
3e-6 of FP64, gradients within about 1e-5 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_band_matches_fp64():
    from oracle.pyadjoint import AdjointOracle
    from sharc.volrus_b200.adjoint import AdvectionFunction
    r, side = 72.0, 20
    c = np.stack(np.unravel_index(np.arange(side ** 3), (side,) * 3), 1)
    c = c[np.abs(np.linalg.norm(c * 8 + 3.5 - 79.7, axis=1) - r) < 11].astype(np.int32)
    loc = np.stack(np.unravel_index(np.arange(512), (8, 8, 8)), 1)
    phi = np.concatenate([np.linalg.norm(q[:, None] * 8 + loc[None] - 79.7, axis=2) - r
                          for q in np.array_split(c, 16)]).astype(np.float32)
    on = np.abs(phi) < 3
    keep = on.any(1)
    o, phi, on = c[keep] * 8, phi[keep].clip(-3, 3), on[keep]
    m = np.packbits(on, axis=1, bitorder="little").view(np.uint64)
    n, cell, K = 43, 4.0, 2
    x, y, z = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    V = np.stack([0.9 * np.sin(0.5 * x + 0.3 * a) * np.cos(0.4 * y + a) * np.cos(0.45 * z - a)
                  for a in range(3)]).astype(np.float32)
    fn = AdvectionFunction(o, np.ascontiguousarray(m), phi, V, cell, 1.0, 50.0, K, 2)
    assert fn.n_band > 2 * 148 * 4 * 8 * 32  # more chunks of up to 32 than two waves hold
    lam = np.random.default_rng(3).standard_normal(fn.n_band).astype(np.float32)
    phik = fn.forward(None, None)
    g0, gv = fn.backward(lam)
    orc = AdjointOracle(o, m, phi.astype(np.float64), 3.0, V.astype(np.float64), n, cell, 1.0, 50.0, 0.0, K)
    assert orc.nb == fn.n_band
    assert np.max(np.abs(phik - orc.forward())) < 2e-5
    r0, rv = orc.backward(lam.astype(np.float64))
    assert np.linalg.norm(g0 - r0) / np.linalg.norm(r0) < 2e-5
    assert np.linalg.norm(gv.reshape(-1) - rv) / np.linalg.norm(rv) < 2e-5
    fn.close()
