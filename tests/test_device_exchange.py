"""Device uploads check their origins and build the index in one round trip,
read-outs are bounded on the device, and the step counter travels with its
launch: every outcome a caller can see, for empty, small and full states."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 96


def ball(n, seed):
    """n distinct leaves around a sphere's surface values (any subset steps)."""
    rng = np.random.default_rng(seed)
    o = np.stack(np.unravel_index(rng.permutation(6 ** 3)[:n], (6, 6, 6)), 1).astype(np.int32) * 8 + 64
    x = o[:, None, :] + np.stack(np.unravel_index(np.arange(512), (8, 8, 8)), 1)[None]
    v = (np.linalg.norm(x - 88.0, axis=2) - 14.0).clip(-3, 3).astype(np.float32)
    m = np.packbits(np.abs(v) < 3, axis=1, bitorder="little").view(np.uint64)
    return o, np.ascontiguousarray(m), v


def level_set(precision):
    from sharc.volrus_b200.method import LevelSet
    return LevelSet.from_leaves(*ball(2, 0), {"kind": "constant", "c": (0.5, 0.25, 0.0)}, 1.0, precision=precision,
                                capacity=CAP)


class Buffers:
    """Device buffers of `cap` records, masks and values starting `skew` bytes
    past an aligned address."""

    def __init__(self, cap, skew=0):
        import torch
        self.cap = cap
        self.raw = [torch.full((max(cap, 1) * b + 16,), 0x5A, dtype=torch.uint8, device="cuda") for b in (12, 64, 2048)]
        self.skew = (0, skew, skew)

    def ptr(self):
        return [r.data_ptr() + s for r, s in zip(self.raw, self.skew)]

    def put(self, arrays):
        import torch
        for r, s, a in zip(self.raw, self.skew, arrays):
            b = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy())
            r[s:s + b.numel()] = b.cuda()
        torch.cuda.synchronize()

    def get(self, n):
        h = [r.cpu().numpy()[s:] for r, s in zip(self.raw, self.skew)]
        return (h[0][:12 * n].copy().view(np.int32).reshape(n, 3), h[1][:64 * n].copy().view(np.uint64).reshape(n, 8),
                h[2][:2048 * n].copy().view(np.float32).reshape(n, 512))


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("precision,skew", [(0, 0), (1, 0), (0, 4), (0, 8), (0, 1), (1, 4)])
@pytest.mark.parametrize("n", [0, 1, 33, CAP])
def test_upload_step_read_out(precision, skew, n):
    o, m, v = ball(n, n) if n else (np.zeros((0, 3), np.int32), np.zeros((0, 8), np.uint64), np.zeros((0, 512), np.float32))
    want = v.astype(np.float16).astype(np.float32) if precision else v
    ls = level_set(precision)
    b = Buffers(n, skew)
    b.put((o, m, v))
    ls.upload_device(*b.ptr(), n)
    out = Buffers(CAP)
    assert ls.download_device(*out.ptr(), CAP) == n and same(out.get(n), (o, m, want))
    if n and n < CAP:  # the index serves steps as a host upload's does
        ls.set_step(3)
        ls.step(1)
        ref = level_set(precision)
        ref.upload(o, m, want)
        ref.set_step(3)
        ref.step(1)
        assert ls.info()[1:] == ref.info()[1:] and same(ls.arrays(), ref.arrays())
        ref.close()
    ls.close()


@pytest.mark.parametrize("cap", [0, 1, 32])
def test_small_buffers_stay_untouched(cap):
    from sharc.volrus_b200._lib import VolrusError
    ls = level_set(0)
    a = ball(33, 1)
    b = Buffers(33)
    b.put(a)
    ls.upload_device(*b.ptr(), 33)
    out = Buffers(33)
    with pytest.raises(VolrusError, match="too small"):
        ls.download_device(*out.ptr(), cap)
    assert all((r.cpu().numpy() == 0x5A).all() for r in out.raw)
    assert ls.download_device(*out.ptr(), 33) == 33 and same(out.get(33), a)
    ls.close()


@pytest.mark.parametrize("fault", ["lattice", "twice", "extent"])
def test_refused_upload_then_a_good_one(fault):
    from sharc.volrus_b200._lib import VolrusError
    ls = level_set(0)
    a = ball(33, 1)
    bad = a[0].copy()
    bad[7] = bad[7] + 1 if fault == "lattice" else bad[6] if fault == "twice" else (1 << 30, 0, 0)
    b = Buffers(33)
    b.put((bad, a[1], a[2]))
    with pytest.raises(VolrusError):
        ls.upload_device(*b.ptr(), 33)
    b.put(a)
    ls.upload_device(*b.ptr(), 33)
    out = Buffers(33)
    assert ls.download_device(*out.ptr(), 33) == 33 and same(out.get(33), a)
    ls.close()


@pytest.mark.parametrize("fault", ["lattice", "twice", "extent"])
def test_refused_upload_leaves_nothing_to_step(fault):
    """Steps are refused until the next complete upload, which steps as in a level set that saw no refusal."""
    from sharc.volrus_b200._lib import ERROR_NAMES, VolrusError
    ls, ref = level_set(0), level_set(0)
    a = ball(33, 33)  # steps within the pool of CAP leaves
    bad = a[0].copy()
    bad[7] = bad[7] + 1 if fault == "lattice" else bad[6] if fault == "twice" else (1 << 30, 0, 0)
    b = Buffers(33)
    b.put((bad, a[1], a[2]))
    with pytest.raises(VolrusError):
        ls.upload_device(*b.ptr(), 33)
    for call in (lambda: ls.step(1), lambda: ls.enqueue(1)):
        with pytest.raises(VolrusError) as e:
            call()
        assert ERROR_NAMES[e.value.code] == "VLR_ERR_INVALID"
    b.put(a)
    for s in (ls, ref):
        s.upload_device(*b.ptr(), 33)
        s.step(1)
    assert same(ls.arrays(), ref.arrays())
    ls.close()
    ref.close()
