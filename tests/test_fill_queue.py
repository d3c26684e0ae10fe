"""New leaves of a chunk of the re-tracking scan around and far beyond the 64 it
fills itself and the 256 keys it queues: isolated leaves, active throughout,
each bring in their 26 neighbours, 6,656 in a chunk of 256.  Leaf set and masks are the FP64 oracle's; every new leaf holds copysign(hw, its owner's value
at the clamped position), bit for bit; a second step works from them.

Bounds: those of the parity tests for a step from a common state."""
import numpy as np
import pytest

from tests.method_compare import bits, compare
from tests.test_method_parity import check

pytestmark = pytest.mark.gpu

HW = 3.0


@pytest.mark.parametrize("precision", [0, 1], ids=["f32", "f16"])
@pytest.mark.parametrize("leaves", [2, 3, 9, 10, 343])
def test_many_new_leaves(oracle, leaves, precision):
    from sharc.volrus_b200.method import LevelSet
    side = 7
    c = np.stack(np.unravel_index(np.arange(side ** 3), (side,) * 3), 1)
    o = (c[:leaves] * 32).astype(np.int32)
    x, y, z = np.stack(np.unravel_index(np.arange(512), (8, 8, 8))).astype(np.float32)
    n = np.arange(len(o), dtype=np.float32)[:, None]
    v = (0.6 * np.sin(0.4 * x + 0.1 * n) + 0.5 * np.cos(0.35 * y - 0.2 * n) + 0.2 * np.sin(0.3 * z + n)).astype(np.float32)
    if precision:
        v = v.astype(np.float16).astype(np.float32)
    m = np.full((len(o), 8), ~np.uint64(0))
    vel = {"kind": "constant", "c": (0.25, -0.125, 0.3)}
    ls = LevelSet.from_leaves(o, m, v, vel, 1.0, half_width=HW, precision=precision, integrator=2, reinit_iters=2,
                              capacity=1 << 14)
    state = (o, m, v)
    for step in range(2):
        mo = oracle.MOGrid.from_arrays(state[0], state[1], state[2].astype(np.float64), HW)
        mo.step(vel, 2, 2, float(step), 1.0)
        ls.step(1)
        state = ls.arrays()
        check(compare(state, mo.arrays(), HW), precision, True)
        if step:
            break
        assert len(state[0]) == 27 * len(o)
        at = {tuple(q): i for i, q in enumerate(state[0].tolist())}
        assert not bits(state[1][[i for q, i in at.items() if any(w % 32 for w in q)]]).any()
        w = np.stack(np.unravel_index(np.arange(512), (8, 8, 8)))
        for d in range(27):
            s = np.array([d // 9 - 1, d // 3 % 3 - 1, d % 3 - 1])
            if not s.any():
                continue
            p = np.clip(w + 8 * s[:, None], 0, 7)
            clamped = p[0] * 64 + p[1] * 8 + p[2]
            for q in o:
                own, new = state[2][at[tuple(q.tolist())]], state[2][at[tuple((q + 8 * s).tolist())]]
                assert np.array_equal(new, np.copysign(np.float32(HW), own[clamped]))
    ls.close()
