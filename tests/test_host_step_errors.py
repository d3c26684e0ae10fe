"""What vlr_ls_step_host reports where the automatic slab count pipelines (2^14
leaves and more) is what the one pass reports, and so is the state it leaves."""
import numpy as np
import pytest

from tests.test_errors import _codes, _sphere
from tests.test_host_slabs import _host_step, _pinned, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def state():
    """About 20,000 leaves in pinned buffers."""
    from sharc.volrus_b200.method import LevelSet, large_sphere_grid
    sph, vel = large_sphere_grid(75, seed=3, extent=1600.0)
    ls = LevelSet.spheres([(sph, vel)], 1.0, half_width=3.0, precision=1, integrator=3, reinit_iters=2)
    inp = tuple(_pinned(a) for a in ls.arrays())
    assert 1 << 14 <= len(inp[0]) < 1 << 18
    yield ls, inp
    ls.close()


def _leave_reach_error(ctx):
    from sharc.volrus_b200.method import curl_noise
    vel = curl_noise(5, 256.0, 0.8, 3)
    vel["domain"] = ((0, 0, 0), (256, 256, 256))  # the sphere reaches negative coordinates
    other = _sphere(ctx, 1, vel=vel, radius=20.0)
    other.enqueue(1)
    return other


def _leave_timeout(ctx):
    other = _sphere(ctx, 1, radius=60.0)  # several chunks in the look-back scan
    ctx.check(ctx.lib.vlr_ctx_set_wait_limit(ctx.handle, 2000), "vlr_ctx_set_wait_limit")
    ctx.check(ctx.lib.vlr_ctx_test_stall(ctx.handle, 1), "vlr_ctx_test_stall")
    try:
        other.enqueue(1)
    finally:
        ctx.check(ctx.lib.vlr_ctx_test_stall(ctx.handle, 0), "vlr_ctx_test_stall")
        ctx.check(ctx.lib.vlr_ctx_set_wait_limit(ctx.handle, 0), "vlr_ctx_set_wait_limit")
    return other


@pytest.mark.parametrize("leave,name", [(_leave_reach_error, "VLR_ERR_REACH"), (_leave_timeout, "VLR_ERR_TIMEOUT")])
def test_error_of_an_earlier_call_is_reported(ctx, state, leave, name):
    """An error that another level set's enqueued step left on the context."""
    from sharc.volrus_b200 import VolrusError
    ls, inp = state
    after = []
    for slabs in (1, 0):
        _host_step(ls, inp, slabs)
        other = leave(ctx)
        with pytest.raises(VolrusError) as e:
            _host_step(ls, inp, slabs)
        assert e.value.code == _codes()[name], slabs
        ctx.check_device()  # reported once
        if name == "VLR_ERR_TIMEOUT":  # the step was abandoned: the state waits for an upload
            with pytest.raises(VolrusError) as e:
                ls.step(1)
            assert e.value.code == _codes()["VLR_ERR_INVALID"]
        else:
            after.append((ls.info(), ls.arrays()))
        other.close()
    for a, b in zip(after, after[1:]):
        assert a[0] == b[0] and _same(a[1], b[1])
    assert _same(_host_step(ls, inp, 0), _host_step(ls, inp, 1))


def test_little_device_memory_takes_the_one_pass(ctx, state):
    """Device memory that holds the one pass's buffers but not the pipeline's."""
    import torch
    from sharc.volrus_b200 import Context
    from sharc.volrus_b200.method import LevelSet, large_sphere_grid
    ls, inp = state
    want = _host_step(ls, inp, 1)
    own = Context()  # its pool holds no memory of other tests
    sph, vel = large_sphere_grid(75, seed=3, extent=1600.0)
    other = LevelSet.spheres([(sph, vel)], 1.0, half_width=3.0, precision=1, integrator=3, reinit_iters=2, ctx=own)
    fill = None
    try:
        _host_step(other, inp, 1)  # the one pass's staging stands
        n = len(inp[0])
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty(free - n * 2048 // 2, dtype=torch.uint8, device="cuda")  # the input's values alone do not fit
        got = _host_step(other, inp, 0)
        del fill
        assert _same(got, want)
    finally:
        fill = None
        torch.cuda.empty_cache()
        other.close()
        own.close()


@pytest.mark.parametrize("width", [1 << 20, (1 << 21) - 2, (1 << 21) - 1, 1 << 21, 1 << 27])
def test_states_as_wide_as_the_hash(ctx, width):
    """Leaves at the corners of a box of `width` leaves an axis (the hash holds 2^21): keys of that box and its
    margin need up to 67 bits, and a wider state is refused as the one pass refuses it."""
    from sharc.volrus_b200 import VolrusError
    from sharc.volrus_b200.method import LevelSet
    lo = -((width + 1) // 2)
    c = np.stack(np.unravel_index(np.arange(8), (2, 2, 2)), 1) * width + lo
    o = (np.concatenate([c, [[0, 0, 0]]])[[0, 1, 2, 3, 8, 4, 5, 6, 7]] * 8).astype(np.int32)
    phi = np.full((9, 8, 8, 8), 3.0, np.float32)
    phi[:, 3:5, 3:5, 3:5] = np.random.default_rng(5).uniform(-2, 2, (9, 2, 2, 2))
    phi = phi.reshape(9, 512)
    m = np.ascontiguousarray(np.packbits(np.abs(phi) < 3, axis=1, bitorder="little")).view(np.uint64)
    ls = LevelSet.from_leaves(o[4:5], m[4:5], phi[4:5], {"kind": "constant", "c": (0.25, -0.5, 0.125)}, 1.0,
                              capacity=256, ctx=ctx)
    inp = tuple(_pinned(a) for a in (o, m, phi))
    res = []
    for slabs in (1, 2):
        try:
            res.append(_host_step(ls, inp, slabs))
        except VolrusError as e:
            res.append(e.code)
    if width < 1 << 21:
        assert len(res[0][0]) == 9 and _same(res[0], res[1])
    else:
        assert res[0] == res[1] == _codes()["VLR_ERR_EXTENT"]
    ls.close()


@pytest.mark.parametrize("dims,steps", [((2, 91, 91), 1), ((3, 74, 74), 1), ((4, 64, 64), 1), ((8, 66, 66), 2),
                                        ((16, 64, 64), 4), ((64, 16, 16), 2)])
def test_states_thin_in_x(ctx, dims, steps):
    """The automatic count steps fewer than twice the leaves (a slab also steps two leaves of x beside it), and gives
    the one pass's result at any count."""
    from sharc.volrus_b200.method import LevelSet
    from tests.test_host_slabs import _out
    c = np.stack(np.unravel_index(np.arange(np.prod(dims)), dims), 1).astype(np.int32) * 8
    p = [(c[:, a:a + 1] + w).astype(np.float32) for a, w in enumerate(np.unravel_index(np.arange(512), (8, 8, 8)))]
    phi = (2.5 * np.sin(0.35 * p[0] + 0.1) * np.cos(0.3 * p[1] + 0.2) * np.cos(0.33 * p[2])).astype(np.float32)
    m = np.ascontiguousarray(np.packbits(np.abs(phi) < 2, axis=1, bitorder="little")).view(np.uint64)
    ls = LevelSet.from_leaves(c, m, phi, {"kind": "constant", "c": (0.5, 0.25, -0.3)}, 1.0, precision=1,
                              capacity=3 * len(c) + 8192, ctx=ctx)
    inp = tuple(_pinned(a) for a in (c, m, phi))
    out = _out(3 * len(c) + 8192)
    want = _host_step(ls, inp, 1, out)
    got = _host_step(ls, inp, 0, out)
    ctx.profile(True)  # counts launches
    try:
        before = ctx.kernel_time("k_m_advect")[1]
        counted = _host_step(ls, inp, 0, out)
        assert ctx.kernel_time("k_m_advect")[1] - before == steps
    finally:
        ctx.profile(False)
    assert _same(want, got) and _same(want, counted)
    assert _same(want, _host_step(ls, inp, 3, out))
    ls.close()


def test_wait_that_runs_out_in_a_slab(ctx, state):
    """A bounded wait of the step gives up: reported, the state lost, and an upload brings it back."""
    from sharc.volrus_b200 import VolrusError
    ls, inp = state
    want = _host_step(ls, inp, 1)
    for slabs in (1, 0):
        ctx.check(ctx.lib.vlr_ctx_set_wait_limit(ctx.handle, 2000), "vlr_ctx_set_wait_limit")
        ctx.check(ctx.lib.vlr_ctx_test_stall(ctx.handle, 1), "vlr_ctx_test_stall")
        try:
            with pytest.raises(VolrusError) as e:
                _host_step(ls, inp, slabs)
            assert e.value.code == _codes()["VLR_ERR_TIMEOUT"]
        finally:
            ctx.check(ctx.lib.vlr_ctx_test_stall(ctx.handle, 0), "vlr_ctx_test_stall")
            ctx.check(ctx.lib.vlr_ctx_set_wait_limit(ctx.handle, 0), "vlr_ctx_set_wait_limit")
        with pytest.raises(VolrusError) as e:
            ls.step(1)
        assert e.value.code == _codes()["VLR_ERR_INVALID"]
        ctx.check_device()
        assert _same(_host_step(ls, inp, slabs), want)
