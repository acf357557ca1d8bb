"""The single-pass scan and sort at the edges of their tiles (4096 elements), over many
tiles, on addresses of 4-byte alignment and in place, against numpy (whole numbers)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4095, 4096, 8192, 8193, 4096 * 33 + 5, 4096 * 700 + 1])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_scan(ctx, n, off):
    a = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)  # wraps modulo 2^32
    buf = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    buf[off:off + n] = torch.from_numpy(a.view(np.int32)).cuda()
    out = torch.full((n + 8,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.dev_exclusive_scan_u32(buf.data_ptr() + 4 * off, out.data_ptr() + 4 * off, n)
    want = np.concatenate([[0], np.cumsum(a.astype(np.uint64))[:-1]]).astype(np.uint64).astype(np.uint32)
    got = out.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[off:off + n], want)
    assert (got[:off] == 0xFFFFFFFF).all() and (got[off + n:] == 0xFFFFFFFF).all()
    ctx.dev_exclusive_scan_u32(buf.data_ptr() + 4 * off, buf.data_ptr() + 4 * off, n)  # in place
    assert np.array_equal(buf.cpu().numpy().view(np.uint32)[off:off + n], want)


@pytest.mark.parametrize("n", [2, 33, 4095, 4096, 4097, 8193, 4096 * 33 + 5, 4096 * 300 + 1])
@pytest.mark.parametrize("begin,end", [(0, 8), (0, 16), (5, 29), (32, 64), (0, 64)])
@pytest.mark.parametrize("kind", ["random", "one digit", "few"])
def test_sort(ctx, n, begin, end, kind):
    rng = np.random.default_rng(n + end)
    k = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, n).astype(np.uint64)
    if kind == "one digit":
        k[:] = np.uint64(0xFFFFFFFFFFFFFFFF)
    elif kind == "few":
        k = k[rng.integers(0, min(n, 5), n)]
    v = np.arange(n, dtype=np.uint32)
    dk, dv = torch.from_numpy(k.view(np.int64)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
    torch.cuda.synchronize()
    ctx.dev_sort_pairs_u64(dk.data_ptr(), dv.data_ptr(), n, begin, end)
    top = min(64, begin + 8 * ((end - begin + 7) // 8))  # whole 8-bit digits
    part = (k >> np.uint64(begin)) & np.uint64((1 << (top - begin)) - 1)
    order = np.argsort(part, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), v[order])
