"""The scan and the sort at sizes where their largest forms run: tiles of
20,480 pairs (above 1,638,400 pairs) around their edges, with digits all alike,
shifted, overlapping and batched arrays; look-back words of 64 bits (from 2^30
pairs); scans in which a block takes more than one tile (above 304 tiles of
8,192 items)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 20480


def u32(t):
    return t.cpu().numpy().view(np.uint32)


def on_gpu(x, shift=0):
    import torch
    t = torch.zeros(x.size + 4, dtype=torch.int32, device="cuda")[shift:shift + x.size]
    t.copy_(torch.from_numpy(x.view(np.int32)))
    return t


def expect(k, v, batch, asc):
    k, v = k.reshape(batch, -1), v.reshape(batch, -1)
    o = np.argsort(k if asc else ~k, axis=1, kind="stable")
    return np.take_along_axis(k, o, 1).reshape(-1), np.take_along_axis(v, o, 1).reshape(-1)


def keys_of(kind, n, rng):
    k = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    return {"random": k, "few": k % 3, "high": k & np.uint32(0xFF000000), "same": np.full(n, 0x80FF0001, np.uint32)}[kind]


@pytest.mark.parametrize("n", [81 * TILE - 1, 81 * TILE, 81 * TILE + 1, 1700003])
@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("kind", ["random", "few", "high", "same"])
def test_sort(gpu_lib, n, asc, kind):
    from mscomplex_gb300.primitives import sort_pairs
    rng = np.random.default_rng(n)
    k, v = keys_of(kind, n, rng), rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    for got, want in zip(sort_pairs(on_gpu(k, n & 1), on_gpu(v, 1 + (n & 1)), ascending=asc), expect(k, v, 1, asc)):
        assert np.array_equal(u32(got), want)


@pytest.mark.parametrize("batch,length", [(81, TILE), (81, TILE + 1), (3, 600001), (1700003, 1)])
@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("kind", ["random", "same"])
def test_sort_arrays(gpu_lib, batch, length, asc, kind):
    from mscomplex_gb300.primitives import sort_pairs
    n = batch * length
    rng = np.random.default_rng(n)
    k, v = keys_of(kind, n, rng), rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    for got, want in zip(sort_pairs(on_gpu(k), on_gpu(v), batch=batch, ascending=asc), expect(k, v, batch, asc)):
        assert np.array_equal(u32(got), want)


@pytest.mark.parametrize("batch,length", [(1, 1700003), (1, 81 * TILE), (5, 340001)])
@pytest.mark.parametrize("asc", [1, 0])
def test_sort_in_place(gpu_lib, batch, length, asc):
    import torch
    n = batch * length
    rng = np.random.default_rng(n)
    k, v = keys_of("random", n, rng) >> 20, np.arange(n, dtype=np.uint32)
    a, b = on_gpu(k), on_gpu(v)
    torch.cuda.synchronize()
    ctx = gpu_lib.default_context()
    p, q = C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())
    assert ctx.lib.dmsc_sort_pairs(ctx.h, p, q, p, q, batch, length, asc, None) == 0
    want = expect(k, v, batch, bool(asc))
    assert np.array_equal(u32(a), want[0]) and np.array_equal(u32(b), want[1])


def test_sort_beyond_30_bits(gpu_lib):
    """Keys of few values, values the places: the pairs come out strictly
    ascending, and each names the place its key came from."""
    import torch
    from mscomplex_gb300.primitives import sort_pairs
    n = 2 ** 30 + 12345
    x = torch.randint(0, 1 << 16, (n,), device="cuda", dtype=torch.int32) * 32749
    k, v = sort_pairs(x, torch.arange(n, device="cuda", dtype=torch.int32))
    for a in range(0, n, 1 << 26):
        b = min(n, a + (1 << 26) + 1)  # (a pair in common with the next part)
        kk, vv = k[a:b].long() & 0xFFFFFFFF, v[a:b].long() & 0xFFFFFFFF
        pair = (kk << 31) | vv
        assert bool((pair[1:] > pair[:-1]).all())
        assert int(vv.max()) < n and bool((x[vv] == k[a:b]).all())


@pytest.mark.parametrize("n", [304 * 8192 - 1, 304 * 8192, 304 * 8192 + 1, 609 * 8192 + 5, 5000011])
@pytest.mark.parametrize("shifts", [(0, 0), (1, 0), (0, 3), (2, 2), "in place", "in place, shifted"])
def test_scan(gpu_lib, n, shifts):
    import torch
    from mscomplex_gb300.primitives import prefix_scan
    x = np.random.default_rng(n).integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    src = on_gpu(x, {"in place": 0, "in place, shifted": 3}.get(shifts) if isinstance(shifts, str) else shifts[0])
    out = src if isinstance(shifts, str) else on_gpu(np.zeros(n, np.uint32), shifts[1])
    tot = torch.zeros(1, dtype=torch.int32, device="cuda")
    prefix_scan(src, out=out, total=tot)
    c = np.cumsum(x.astype(np.uint64))
    assert np.array_equal(u32(out), (c - x).astype(np.uint32)) and int(u32(tot)[0]) == int(c[-1] & 0xFFFFFFFF)
