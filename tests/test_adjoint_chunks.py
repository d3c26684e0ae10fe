"""The adjoint's chunked kernels at their edges: leaves of 1 to 512 band voxels
(chunks of up to 32), absent neighbours, one foot offset per neighbourhood
(no candidate test) and several, reach 1 and 2, the windowed and the quad
transpose, and a new velocity in the same plan; against the FP64 oracle.

Three steps of FP32 arithmetic on |phi| <= 3: a blend rounds about 8 times, so
phi_K is within 3 * 8 * 3 * 2^-24 = 4e-6 of FP64, a gradient (sums of 8 terms a
step, weights rounded to 2^-24 of offsets below 2) within about 1e-5 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = (1, 31, 32, 33, 64, 65, 511, 512)


def grid(seed):
    rng = np.random.default_rng(seed)
    cells = np.stack(np.meshgrid(*[np.arange(1, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    o = cells[rng.permutation(27)[:18]]
    o = o[np.lexsort((o[:, 2], o[:, 1], o[:, 0]))].astype(np.int32) * 8
    m = np.zeros((len(o), 8), np.uint64)
    for i in range(len(o)):
        on = np.zeros(512, bool)
        on[rng.permutation(512)[:COUNTS[i % len(COUNTS)]]] = True
        m[i] = np.packbits(on, bitorder="little").view(np.uint64)
    pos = o[:, None, :] + np.stack(np.unravel_index(np.arange(512), (8, 8, 8)), -1)[None]
    p = 2.5 * np.sin(0.31 * pos[..., 0] + 0.7) * np.cos(0.23 * pos[..., 1]) + 0.4 * np.sin(0.4 * pos[..., 2])
    return o, m, p.astype(np.float32)


def field(kind, n, amp, seed):
    rng = np.random.default_rng(seed)
    if kind == "constant":
        u = np.array([0.63, -0.41, 0.27]) * amp
        return np.broadcast_to(u[:, None, None, None], (3, n, n, n)).astype(np.float32)
    x, y, z = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    ph = rng.uniform(0, 6, 9)
    return np.stack([amp * 0.9 * np.sin(0.5 * x + ph[a]) * np.cos(0.4 * y + ph[3 + a]) * np.cos(0.45 * z + ph[6 + a])
                     for a in range(3)]).astype(np.float32)


@pytest.mark.parametrize("kind", ["constant", "smooth"])
@pytest.mark.parametrize("amp,mode", [(1.0, 1), (1.0, 2), (1.0, 0), (1.9, 0)])
def test_chunks_match_fp64(kind, amp, mode):
    from oracle.pyadjoint import AdjointOracle
    from sharc.volrus_b200.adjoint import AdvectionFunction
    o, m, p = grid(5)
    n, cell, dt, K = 17, 2.0, 1.0, 3
    V = field(kind, n, amp, 1)
    fn = AdvectionFunction(o, m, p, V, cell, dt, 50.0, K, 2)
    fn.set_gather(mode)
    rng = np.random.default_rng(9)
    lam = rng.standard_normal(fn.n_band).astype(np.float32)
    for seed in (1, 2):  # the plan's own velocity, then another one in the same plan
        W = field(kind, n, amp * (1.0 if seed == 1 else 0.7), seed)
        phik = fn.forward(None, None if seed == 1 else W)
        g0, gv = fn.backward(lam)
        orc = AdjointOracle(o, m, p.astype(np.float64), 3.0, W.astype(np.float64), n, cell, dt, 50.0, 0.0, K)
        assert orc.nb == fn.n_band
        assert np.max(np.abs(phik - orc.forward())) < 2e-5
        r0, rv = orc.backward(lam.astype(np.float64))
        assert np.linalg.norm(g0 - r0) / np.linalg.norm(r0) < 2e-5
        assert np.linalg.norm(gv.reshape(-1) - rv) / np.linalg.norm(rv) < 2e-5
        again = fn.backward(lam)
        assert np.array_equal(g0, again[0]) and np.array_equal(gv, again[1])
    fn.close()
