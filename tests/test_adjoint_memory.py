"""Memory of the staggered adjoint: the interval of its checkpoints is a wish
that changes no result and asks for no more than the steps can use, and what
creation needs for a while goes back to the device."""
import numpy as np
import pytest

from tests.test_adjoint_order import _sphere_leaves

pytestmark = pytest.mark.gpu

CENTER = (96.0, 96.0, 97.3)


def _field():
    return (np.random.default_rng(2).uniform(-0.8, 0.8, (3, 28, 28, 28))).astype(np.float32)


def _pass(steps, every, r=12.4):
    from sharc.volrus_b200.adjoint import AdvectionFunction
    fn = AdvectionFunction(*_sphere_leaves(CENTER, r), _field(), 8.0, 1.0, 300.0, steps, every)
    phik = fn.forward()
    g0, gv = fn.backward(np.random.default_rng(3).standard_normal(fn.n_band).astype(np.float32))
    fn.close()
    return phik, g0, gv


@pytest.mark.parametrize("steps,intervals", [(1, (1, 2)), (10, (1, 3, 9, 10, 11)), (130, (1, 11, 40, 41, 48, 129, 130, 500))])
def test_any_interval_gives_the_same_bits(steps, intervals):
    ref = _pass(steps, intervals[0])
    assert np.abs(ref[2]).max() > 0
    for every in intervals[1:]:
        for a, b in zip(ref, _pass(steps, every)):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), every


def test_interval_past_the_steps():
    """An interval whose segment of gradients would not fit the device (of values, it would)."""
    ref = _pass(10, 3)
    for a, b in zip(ref, _pass(10, 1_500_000)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_creation_gives_its_temporaries_back():
    """About 390,000 band voxels: 225 MB of sort buffers."""
    import torch
    from sharc.volrus_b200 import Context
    from sharc.volrus_b200.adjoint import AdvectionFunction
    _pass(2, 2)  # kernels and libraries are in place
    leaves = _sphere_leaves(CENTER, 72.0)
    ctx = Context()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    fn = AdvectionFunction(*leaves, _field(), 8.0, 1.0, 300.0, 4, 2, ctx=ctx)
    assert fn.n_band * 576 > 200 << 20
    fn.forward()
    fn.backward(np.ones(fn.n_band, np.float32))
    fn.close()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 100 << 20
    ctx.close()
