"""The gradient and label tiles with their neighbours on every side: interior
tiles, tiles cut to a column or a row, paths that wind through a whole tile,
equal heights in every position, both vertex orders.  Cells, owners and the
complex are compared with the oracle's, exactly."""
import numpy as np
import pytest

from helpers import assert_same_complex, full_rect, tie_field

pytestmark = pytest.mark.gpu


def spiral(ny, nx):
    """One path down a spiral trench between walls, through every tile."""
    f = np.full((ny, nx), 2.0, np.float32)
    y, x, dy, dx = 0, 0, 0, 1
    for k in range(ny * nx):
        f[y, x] = 1.0 - k / (ny * nx)
        for _ in range(2):
            ay, ax, by, bx = y + dy, x + dx, y + 2 * dy, x + 2 * dx
            free = 0 <= ay < ny and 0 <= ax < nx and f[ay, ax] == 2.0
            if free and not (0 <= by < ny and 0 <= bx < nx and f[by, bx] != 2.0):
                break
            dy, dx = dx, -dy
        else:
            break
        y, x = ay, ax
    return f


def field_of(kind, ny, nx):
    if kind == "spiral":
        return spiral(ny, nx)
    if kind == "infinite":
        f = tie_field(ny, nx, 5, ny + nx)
        f[f == f.max()], f[f == f.min()] = np.inf, -np.inf
        f[::3, ::2] *= np.float32(-0.0)
        return np.nan_to_num(f, nan=0.0, posinf=np.inf, neginf=-np.inf)
    return tie_field(ny, nx, {"two levels": 2, "many levels": 4000}[kind], ny * nx)


@pytest.mark.parametrize("order", ["ascending", "descending"])
@pytest.mark.parametrize("kind", ["two levels", "many levels", "infinite", "spiral"])
@pytest.mark.parametrize("ny,nx", [(196, 259), (193, 257), (260, 194), (66, 66)])
def test_tiles(gpu_lib, oracle, ny, nx, kind, order):
    f = field_of(kind, ny, nx)
    r = full_rect(f)
    what = f"{kind} {nx}x{ny} {order}"
    g = gpu_lib.GridDataset(r, r).init(f)
    if order == "descending":
        o, g = oracle.Dataset(f, r, r, mode=oracle.MODE_OCL), g.work_ocl()
    else:
        o, g = oracle.Dataset(f, r, r), g.work()
    for name, a, b in zip(("flags", "pairs", "own"), g.cells(), o.cells()):
        assert np.array_equal(a, b), f"{what}: {name} differs at {np.argwhere(a != b)[:5].tolist()}"
    got, want = g.writeout_connectivity().export(), o.msc()
    nan = np.isnan(want["fn"])  # edges between both infinities; the bits of a NaN are the machine's
    assert np.array_equal(np.isnan(got["fn"]), nan), what
    got["fn"] = np.where(nan, np.float32(0), got["fn"])
    want["fn"] = np.where(nan, np.float32(0), want["fn"])
    assert_same_complex(got, want, what)
