"""The merges' boundary steps by several warps (merge_up's cancellations in the
loop's order, merge_down's uncancellations side by side) where they change
over: boundaries around a multiple of 32 cells, lists of one lane, one warp
and longer, pairs with both points on the boundary.  Every node of the piece
tree against the oracle's, exactly."""
import numpy as np
import pytest

from helpers import assert_same_complex, tie_field

pytestmark = pytest.mark.gpu

GRAPH = ("rect_ext", "cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")


def check(M, oracle, f, levels, split2d, what, tresh=0.0):
    ctx = M.Context()
    ctx.set_merge_parallel_min(0)
    want = oracle.Pipeline(f, levels=levels, tresh=tresh, split2d=split2d)
    got = M.GridDataManager(f, levels=levels, tresh=tresh, split2d=split2d, ctx=ctx)
    for i in range(2 * got.num_pieces - 1):
        assert_same_complex(got.piece(i).export(), want.piece(i), f"{what} node {i}", keys=GRAPH)
    del got
    ctx.close()


@pytest.mark.parametrize("nx", [5, 16, 17, 33, 65, 130])
@pytest.mark.parametrize("levels", [1, 3])
def test_boundary_lengths(gpu_lib, oracle, nx, levels):
    f = np.random.default_rng(nx).random((64, nx), dtype=np.float32)
    check(gpu_lib, oracle, f, levels, False, f"{nx} wide, {levels} levels")


def basin(n, pits, seed):
    """A basin floor with `pits` pits and peaks: the floor's lists grow to
    hundreds of runs over the merges."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:n, 0:n]
    f = 0.01 * np.hypot(x - n / 2, y - n / 2) / n + rng.uniform(0, 1e-6, (n, n))
    i = rng.integers(1, n - 1, pits), rng.integers(1, n - 1, pits)
    f[i] += np.where(rng.random(pits) < 0.2, -0.5, 0.5)
    return f.astype(np.float32)


@pytest.mark.parametrize("pits", [20, 200, 900])
@pytest.mark.parametrize("split2d", [False, True])
def test_long_lists(gpu_lib, oracle, pits, split2d):
    check(gpu_lib, oracle, basin(96, pits, pits), 2, split2d, f"{pits} pits")


@pytest.mark.parametrize("seed", range(3))
def test_flat_boundaries(gpu_lib, oracle, seed):
    """Two or three heights: most boundary cells pair along the boundary."""
    check(gpu_lib, oracle, tie_field(48, 52, 2 + seed % 2, seed), 3, True, f"flat {seed}", tresh=0.1)
