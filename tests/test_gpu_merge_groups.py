"""merge_up's boundary cells in groups that meet at no point: many groups (white
noise), one group (an extremum that all cells share), a few of each, boundaries
from one cell group to thousands of cells, several merges a level.  Every node
of the piece tree against the oracle's, exactly."""
import numpy as np
import pytest

from helpers import assert_same_complex, tie_field

pytestmark = pytest.mark.gpu

GRAPH = ("rect_ext", "cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")


def field_of(kind, ny, nx):
    rng = np.random.default_rng(ny * nx)
    f = rng.random((ny, nx)).astype(np.float32)
    if kind == "noise":
        return f
    if kind == "one basin":  # every boundary point drains to the same minimum
        y, x = np.mgrid[0:ny, 0:nx]
        return (np.hypot(x - nx / 2, y - ny / 2) + 1e-3 * f).astype(np.float32)
    if kind == "noise beside a slope":
        f[:, nx // 2:] = np.arange(nx - nx // 2, dtype=np.float32) + 2 + 1e-3 * f[:, nx // 2:]
        return f
    return tie_field(ny, nx, 3, nx)


@pytest.mark.parametrize("kind", ["noise", "one basin", "noise beside a slope", "ties"])
@pytest.mark.parametrize("ny,nx,levels,split2d", [(9, 300, 1, False), (200, 600, 3, True), (40, 3, 2, False)])
def test_groups(gpu_lib, oracle, kind, ny, nx, levels, split2d):
    f = field_of(kind, ny, nx)
    ctx = gpu_lib.Context()
    ctx.set_merge_parallel_min(0)
    want = oracle.Pipeline(f, levels=levels, tresh=0.0, split2d=split2d)
    got = gpu_lib.GridDataManager(f, levels=levels, tresh=0.0, split2d=split2d, ctx=ctx)
    for i in range(2 * got.num_pieces - 1):
        assert_same_complex(got.piece(i).export(), want.piece(i), f"{kind} {nx}x{ny} node {i}", keys=GRAPH)
    del got
    ctx.close()


@pytest.mark.parametrize("up", [True, False])
@pytest.mark.parametrize("n", [301, 421])
def test_a_boundary_point_with_thousands_of_saddles(gpu_lib, oracle, n, up):
    """A funnel of peaks drains to one point of the shared boundary, which pairs
    across it: cancelling it moves more values than a warp's scratch holds."""
    y, x = np.mgrid[0:n, 0:n].astype(np.float64)
    row = n // 2
    far = np.hypot(x - n // 2, y - row)
    side = y >= row if up else y <= row
    f = np.where(side, far, -far - 1.0)
    f[row, :] = far[row, :]
    f[side & (y % 3 == 0) & (x % 3 == 1) & (np.abs(y - row) > 1)] += 9.0
    f = f.astype(np.float32)
    want = oracle.Pipeline(f, levels=1, tresh=0.0, split2d=False)
    assert np.diff(want.piece(2)["asc_off"]).max() > 5000
    got = gpu_lib.GridDataManager(f, levels=1, tresh=0.0, split2d=False)
    for i in range(3):
        assert_same_complex(got.piece(i).export(), want.piece(i), f"funnel {n} node {i}", keys=GRAPH)
