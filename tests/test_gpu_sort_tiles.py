"""The sort where its tiles change: one block with 4 or 8 pairs a thread, tiles of
4,096 and of 20,480 pairs, alone and in batches, against a stable host sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n", [(1, 4095), (1, 4096), (1, 4097), (1, 8191), (1, 8192), (1, 8193), (1, 12289),
                                     (1, 1638400), (1, 1638401), (3, 1365), (3, 2731), (257, 32), (700, 2341)])
@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("keys", ["random", "few"])
def test_tiles(gpu_lib, batch, n, asc, keys):
    import torch
    from mscomplex_gb300.primitives import sort_pairs
    rng = np.random.default_rng(batch * n)
    k = rng.integers(0, 5 if keys == "few" else 2 ** 32, size=batch * n, dtype=np.uint64).astype(np.uint32)
    v = rng.integers(0, 2 ** 32, size=batch * n, dtype=np.uint64).astype(np.uint32)
    ok, ov = sort_pairs(torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda(), batch=batch, ascending=asc)
    o = np.argsort((k if asc else ~k).reshape(batch, n), axis=1, kind="stable")
    assert np.array_equal(ok.cpu().numpy().view(np.uint32), np.take_along_axis(k.reshape(batch, n), o, 1).reshape(-1))
    assert np.array_equal(ov.cpu().numpy().view(np.uint32), np.take_along_axis(v.reshape(batch, n), o, 1).reshape(-1))
