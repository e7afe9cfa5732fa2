"""The scan and the sort around the edges of their tiles (8,192 items; 20,480
pairs), on unaligned and overlapping arrays, and on digits that are all alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scan(x, shift_in=0, shift_out=0):
    import torch
    from mscomplex_gb300.primitives import prefix_scan
    n = x.size
    src = torch.zeros(n + 4, dtype=torch.int32, device="cuda")[shift_in:shift_in + n]
    src.copy_(torch.from_numpy(x.view(np.int32)))
    out = torch.zeros(n + 4, dtype=torch.int32, device="cuda")[shift_out:shift_out + n]
    tot = torch.zeros(1, dtype=torch.int32, device="cuda")
    prefix_scan(src, out=out, total=tot)
    return out.cpu().numpy().view(np.uint32), int(tot.cpu().numpy().view(np.uint32)[0])


@pytest.mark.parametrize("n", [1, 3, 127, 129, 511, 513, 8191, 8192, 8193, 16385, 300007])
@pytest.mark.parametrize("shifts", [(0, 0), (1, 0), (0, 3)])
def test_scan_tiles(gpu_lib, n, shifts):
    x = np.random.default_rng(n).integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    got, tot = scan(x, *shifts)
    c = np.cumsum(x.astype(np.uint64))
    assert np.array_equal(got, (c - x).astype(np.uint32)) and tot == int(c[-1] & 0xFFFFFFFF)


def sort(k, v, batch, asc, shift=0):
    import torch
    from mscomplex_gb300.primitives import sort_pairs
    t = torch.zeros(2, k.size + 1, dtype=torch.int32, device="cuda")
    a, b = t[0][shift:shift + k.size], t[1][shift:shift + k.size]
    a.copy_(torch.from_numpy(k.view(np.int32)))
    b.copy_(torch.from_numpy(v.view(np.int32)))
    ok, ov = sort_pairs(a, b, batch=batch, ascending=asc)
    return ok.cpu().numpy().view(np.uint32), ov.cpu().numpy().view(np.uint32)


def expect(k, v, batch, asc):
    ks, vs = [], []
    for kk, vv in zip(k.reshape(batch, -1), v.reshape(batch, -1)):
        o = np.argsort(kk if asc else ~kk, kind="stable")
        ks.append(kk[o])
        vs.append(vv[o])
    return np.concatenate(ks), np.concatenate(vs)


@pytest.mark.parametrize("n", [2, 31, 33, 511, 513, 20479, 20480, 20481, 40961, 200003])
@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("keys", ["random", "few", "high", "same"])
def test_sort_tiles(gpu_lib, n, asc, keys):
    rng = np.random.default_rng(n)
    k = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    k = {"random": k, "few": k % 3, "high": k & np.uint32(0xFF000000), "same": np.full(n, 0xFFFFFFFF, np.uint32)}[keys]
    v = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    for got, want in zip(sort(k, v, 1, asc, shift=n & 1), expect(k, v, 1, asc)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("batch,length", [(2, 3), (20480, 1), (5, 4096), (5, 4097), (300, 77), (70000, 3), (17, 20001)])
@pytest.mark.parametrize("asc", [True, False])
def test_sort_arrays(gpu_lib, batch, length, asc):
    rng = np.random.default_rng(batch + length)
    k = (rng.integers(0, 2 ** 32, size=batch * length, dtype=np.uint64) >> 20).astype(np.uint32)
    v = rng.integers(0, 2 ** 32, size=batch * length, dtype=np.uint64).astype(np.uint32)
    for got, want in zip(sort(k, v, batch, asc), expect(k, v, batch, asc)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("batch,length", [(1, 5000), (1, 50000), (5, 700), (5, 9000)])
def test_sort_in_place(gpu_lib, batch, length):
    """Output arrays that are the inputs, as the C entry point takes them."""
    import ctypes as C
    import torch
    n = batch * length
    rng = np.random.default_rng(n)
    k = (rng.integers(0, 2 ** 32, size=n, dtype=np.uint64) >> 22).astype(np.uint32)
    v = np.arange(n, dtype=np.uint32)
    a, b = (torch.from_numpy(x.view(np.int32)).cuda() for x in (k, v))
    torch.cuda.synchronize()
    ctx = gpu_lib.default_context()
    rc = ctx.lib.dmsc_sort_pairs(ctx.h, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(a.data_ptr()),
                                 C.c_void_p(b.data_ptr()), batch, length, 1, None)
    assert rc == 0
    want = expect(k, v, batch, True)
    assert np.array_equal(a.cpu().numpy().view(np.uint32), want[0])
    assert np.array_equal(b.cpu().numpy().view(np.uint32), want[1])
