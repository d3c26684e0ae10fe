"""Device-resident uploads and downloads move whole leaves exactly, from and
into device buffers of any 4-byte alignment (the vector path needs 16 bytes,
the scalar path serves the rest), for leaf counts around a CTA's eight warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def leaves(n, seed):
    rng = np.random.default_rng(seed)
    o = np.stack(np.unravel_index(rng.permutation(16 ** 3)[:n], (16, 16, 16)), 1).astype(np.int32) * 8
    m = rng.integers(0, 2 ** 64, (n, 8), dtype=np.uint64)
    v = rng.uniform(-3, 3, (n, 512)).astype(np.float32)
    return o, m, v


@pytest.mark.parametrize("precision", [0, 1], ids=["f32", "f16"])
@pytest.mark.parametrize("shift_in,shift_out", [(0, 0), (1, 0), (0, 2), (3, 1)])
@pytest.mark.parametrize("n", [1, 8, 9, 300])
def test_round_trip_any_alignment(precision, shift_in, shift_out, n):
    import torch
    from sharc.volrus_b200.method import LevelSet
    o, m, v = leaves(n, n)
    ls = LevelSet.from_leaves(o[:1], m[:1], v[:1], {"kind": "constant", "c": (0.0, 0.0, 0.0)}, 1.0,
                              precision=precision, capacity=512)
    dev = torch.device("cuda")
    d_o, d_m = torch.from_numpy(o).to(dev), torch.from_numpy(m.view(np.int64)).to(dev)
    d_in = torch.zeros(n * 512 + shift_in, device=dev)
    d_in[shift_in:] = torch.from_numpy(v).to(dev).reshape(-1)
    torch.cuda.synchronize()
    ls.upload_device(d_o.data_ptr(), d_m.data_ptr(), d_in.data_ptr() + 4 * shift_in, n)
    o2, m2 = torch.zeros_like(d_o), torch.zeros_like(d_m)
    out = torch.full((n * 512 + shift_out + 8,), 7.0, device=dev)
    torch.cuda.synchronize()
    assert ls.download_device(o2.data_ptr(), m2.data_ptr(), out.data_ptr() + 4 * shift_out, n) == n
    want = v.astype(np.float16).astype(np.float32) if precision else v
    assert torch.equal(o2, d_o) and torch.equal(m2, d_m)
    got = out.cpu().numpy()
    assert np.array_equal(got[shift_out:shift_out + n * 512].reshape(n, 512), want)
    assert np.all(got[:shift_out] == 7.0) and np.all(got[shift_out + n * 512:] == 7.0)
    so, sm, sv = ls.arrays()  # the sorted host download of the same pool
    order = np.lexsort((o[:, 2], o[:, 1], o[:, 0]))
    assert np.array_equal(so, o[order]) and np.array_equal(sm, m[order]) and np.array_equal(sv, want[order])
    ls.close()
