"""The reinitialisation kernel against a dense f32 restatement on random
fields: every voxel of the leaf box, leaves with absent neighbours on any
side, sparse to full activity, zero and signed-zero values, both modes and
value types.  The velocity is zero, so the step is reinitialisation alone.

Bounds: the restatement rounds as the kernel does except for the reciprocal
root (2^-22 relative); an update is 0.5 s (G - 1) with |G| < 13 for values
within 3.5, so one iteration differs by less than 0.5 * 14 * 2^-22 < 2e-6 plus
rounding, and the second, whose G moves by at most 2 sqrt(3) times that, by
less than 1e-5.  f16 results add half a unit of the last place below 4, 1e-3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HW = np.float32(3.0)
AXES = ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))


def neighbours(phi, centre):
    """The six neighbours, copysign(hw, centre) where the leaf is absent (NaN)."""
    out = []
    for a in AXES:
        n = np.roll(phi, [-s for s in a], (0, 1, 2))
        out.append(np.where(np.isnan(n), np.copysign(HW, centre), n))
    return out


def godunov(p, n, s):
    sg = np.where(s >= 0, np.float32(1), np.float32(-1))
    g = np.float32(0)
    for a in range(3):
        u = np.maximum(np.maximum(sg * (p - n[2 * a]), sg * (p - n[2 * a + 1])), np.float32(0))
        g = g + u * u
    return p - np.float32(0.5) * s * (np.sqrt(g) - np.float32(1))


def reinit(phi1, D, iters, fix):
    s = (phi1 / np.sqrt(phi1.astype(np.float64) ** 2 + 1)).astype(np.float32)
    d = np.full_like(phi1, np.nan)
    if fix:
        n = neighbours(phi1, phi1)
        cut = np.zeros(phi1.shape, bool)
        g = np.float32(0)
        for q in n:
            cut |= phi1 * q < 0
        for a in range(3):
            xp, xm = n[2 * a], n[2 * a + 1]
            m = np.maximum(np.maximum(np.abs(xp - xm) * np.float32(0.5), np.abs(xp - phi1)),
                           np.maximum(np.abs(phi1 - xm), np.float32(1e-6)))
            g = g + m * m
        d = np.where(cut, phi1 / np.sqrt(g), np.nan).astype(np.float32)
    cur = phi1
    for _ in range(iters):
        new = godunov(cur, neighbours(cur, cur), s)
        relax = cur - np.float32(0.5) * (np.copysign(np.abs(cur), phi1) - d)
        cur = np.where(D, np.where(np.isnan(d), new, relax), cur)
    return cur


@pytest.mark.parametrize("precision", [0, 1], ids=["f32", "f16"])
@pytest.mark.parametrize("iters,fix", [(0, 0), (1, 0), (2, 0), (1, 1), (2, 1)])
@pytest.mark.parametrize("n,density", [(1, 0.5), (27, 1.0), (40, 0.02), (40, 0.4)])
def test_against_dense(precision, iters, fix, n, density):
    from sharc.volrus_b200.method import LevelSet
    rng = np.random.default_rng(1000 * n + int(100 * density) + 10 * iters + fix)
    side = {1: 1, 27: 3, 40: 4}[n]
    c = np.stack(np.unravel_index(rng.permutation(side ** 3)[:n], (side,) * 3), 1)
    o = (c * 8).astype(np.int32)
    v = rng.uniform(-3.5, 3.5, (n, 512)).astype(np.float32)
    v[rng.random((n, 512)) < 0.05] = 0.0
    v[rng.random((n, 512)) < 0.05] *= -0.0
    if precision:
        v = v.astype(np.float16).astype(np.float32)
    act = rng.random((n, 512)) < density
    act[0, 100] = True
    m = np.packbits(act, axis=1, bitorder="little").view(np.uint64)
    size = (side + 2) * 8
    phi = np.full((size,) * 3, np.nan, np.float32)
    on = np.zeros((size,) * 3, bool)
    for i in range(n):
        w = tuple(slice(8 * (q + 1), 8 * (q + 2)) for q in c[i])
        phi[w] = v[i].reshape(8, 8, 8)
        on[w] = act[i].reshape(8, 8, 8)
    D = on.copy()
    for a in range(3):
        D = D | np.roll(D, 1, a) | np.roll(D, -1, a)
    D &= ~np.isnan(phi)
    with np.errstate(invalid="ignore"):
        want = reinit(np.where(D | np.isnan(phi), phi, np.copysign(HW, phi)), D, iters, fix)
    ls = LevelSet.from_leaves(o, np.ascontiguousarray(m), v, {"kind": "constant", "c": (0.0, 0.0, 0.0)}, 1.0,
                              precision=precision, capacity=512, integrator=1, reinit_iters=iters, reinit_mode=fix)
    ls.step(1)
    so, sm, sv = ls.arrays()
    ls.close()
    tol = 1e-5 + (1e-3 if precision else 0.0)
    got = {tuple(q): i for i, q in enumerate(so.tolist())}
    for i in range(n):
        w = tuple(slice(8 * (q + 1), 8 * (q + 2)) for q in c[i])
        ref, inside = want[w].reshape(512), D[w].reshape(512)
        ref_on = inside & (np.abs(ref) < HW)
        ref_v = np.where(ref_on, ref, np.copysign(HW, ref))
        k = got.get(tuple(o[i].tolist()))
        if k is None:
            assert not (inside & (np.abs(ref) < HW - tol)).any()
            continue
        bits = np.unpackbits(sm[k].view(np.uint8), bitorder="little").astype(bool)
        assert (np.abs(np.abs(ref[bits ^ ref_on]) - HW) < tol).all()
        assert (np.abs(sv[k] - ref_v) <= tol).all()
