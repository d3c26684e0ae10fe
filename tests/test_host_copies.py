"""Copies between pageable arrays and the device pass through pinned chunks in
parts: the bytes of every size around a part, a chunk and the ring arrive, both
ways, and what lies beside them stays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("nbytes", [24, 3 * MB - 24, 3 * MB, 3 * MB + 24, 4 * MB + MB // 2 + 24, 6 * MB, 8 * MB + 24,
                                    10 * MB - 24, 33 * MB + 264])
def test_positions_there_and_back(nbytes):
    """A zero velocity returns the positions: both directions, in place."""
    from sharc.volrus_b200 import _lib
    from sharc.volrus_b200.tools import _as_device, make_uniform_velocity
    import ctypes as C
    n = nbytes // 24
    vel = make_uniform_velocity(1.0, (0.0, 0.0, 0.0))
    ctx = _lib.Context.default()
    rng = np.random.default_rng(nbytes)
    buf = rng.uniform(-8, 8, 3 * n + 8)
    want = buf.copy()
    p = buf[4:4 + 3 * n]
    g = [_as_device(v, ctx)[0] for v in (vel.vx, vel.vy, vel.vz)]
    ctx.check(ctx.lib.vlr_advect_particles(ctx.handle, g[0].handle, g[1].handle, g[2].handle,
                                           _lib.ptr(p, C.c_double), n, 0.5, 0), "vlr_advect_particles")
    assert np.array_equal(buf, want)


@pytest.mark.parametrize("n", [1, 56174, 56173, 150000])
def test_points_into_a_second_array(n):
    """In place and into a second array agree; the given particles stay."""
    from sharc.volrus_b200 import _lib
    from sharc.volrus_b200.points import PARTICLE, PointDataGrid
    from sharc.volrus_b200.tools import _as_device, make_uniform_velocity
    import ctypes as C
    vel = make_uniform_velocity(1.0, (0.75, -0.5, 0.25))
    ctx = _lib.Context.default()
    rng = np.random.default_rng(n)
    a = np.zeros(n, PARTICLE)
    a["position"] = rng.uniform(-24, 24, (n, 3))
    a["velocity"] = rng.normal(size=(n, 3))
    a["id"] = np.arange(n)
    keep, out, inplace = a.copy(), np.empty(n, PARTICLE), a.copy()
    grids = [_as_device(v, ctx)[0] for v in (vel.vx, vel.vy, vel.vz)]
    g = [d.handle for d in grids]
    inv = PointDataGrid(1.0).inverse_rows()
    res = []
    for src, dst in ((a, out), (inplace, None)):
        org, start, k = np.zeros((n, 3), np.int32), np.zeros(n + 1, np.uint32), C.c_size_t()
        head = (ctx.handle, *g, _lib.ptr(inv, C.c_double), src.ctypes.data_as(C.c_void_p))
        tail = (n, 0.5, 1, _lib.ptr(org, C.c_int32), _lib.ptr(start, C.c_uint32), n, C.byref(k))
        if dst is None:
            ctx.check(ctx.lib.vlr_advect_points(*head, *tail), "vlr_advect_points")
        else:
            ctx.check(ctx.lib.vlr_advect_points_to(*head, dst.ctypes.data_as(C.c_void_p), *tail), "vlr_advect_points_to")
        res.append((org[:k.value].copy(), start[:k.value + 1].copy()))
    assert a.tobytes() == keep.tobytes() and out.tobytes() == inplace.tobytes()
    assert all(np.array_equal(x, y) for x, y in zip(*res))


def test_contexts_side_by_side():
    """Each context copies with threads of its own, and leaves them behind when it goes."""
    import threading
    from sharc.volrus_b200._lib import Context
    from sharc.volrus_b200.tools import advect_particles_euler, make_uniform_velocity
    want = {s: np.random.default_rng(s).uniform(-8, 8, (200000, 3)) for s in range(3)}
    got = {}

    def run(s):
        for _ in range(3):
            ctx = Context()
            got[s] = advect_particles_euler(want[s], make_uniform_velocity(1.0, (0.0, 0.0, 0.0)), 0.5, ctx=ctx)
            ctx.close()
    ts = [threading.Thread(target=run, args=(s,)) for s in want]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert all(np.array_equal(got[s], want[s]) for s in want)


def test_threads_end_with_their_context():
    """The threads of large copies start with a context's first one and are joined by its destruction."""
    import os
    import time
    from sharc.volrus_b200._lib import Context
    from sharc.volrus_b200.tools import advect_particles_euler, make_uniform_velocity

    def names():
        n = 0
        for t in os.listdir("/proc/self/task"):
            try:
                n += open(f"/proc/self/task/{t}/comm").read().strip() == "vlr-copy"
            except OSError:
                pass  # gone since the listing
        return n
    vel = make_uniform_velocity(1.0, (0.0, 0.0, 0.0))
    pos = np.random.default_rng(0).uniform(-8, 8, (200000, 3))
    base = names()
    ctx = Context()
    advect_particles_euler(pos[:1000], vel, 0.5, ctx=ctx)
    assert names() == base
    for _ in range(2):
        advect_particles_euler(pos, vel, 0.5, ctx=ctx)
        assert names() == base + 3
    ctx.close()
    until = time.monotonic() + 1.0  # the system may list a joined thread for an instant
    while names() != base and time.monotonic() < until:
        time.sleep(0.001)
    assert names() == base
