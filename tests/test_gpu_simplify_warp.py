"""The simplification's warp-wide replay where its parts change over: heaps
around the shared-memory levels, neighbour lists around a register, a lane and
a warp, batches past one complex per SM, values that are not finite.  Every
complex is compared with the oracle's, exactly."""
import numpy as np
import pytest

from helpers import assert_same_complex, full_rect, smooth_field, tie_field

pytestmark = pytest.mark.gpu

GRAPH = ("cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")


def simplified(M, oracle, f, tresh, what):
    r = full_rect(f)
    want = oracle.Dataset(f, r, r, tresh=tresh).msc()
    m = M.GridDataset(r, r).init(f).work().writeout_connectivity()
    st = m.simplify_un_simplify(tresh)
    assert_same_complex(m.export(), want, what)
    return st


@pytest.mark.parametrize("ny,nx", [(2, 2), (2, 9), (3, 3), (5, 4), (7, 31), (17, 17)])
@pytest.mark.parametrize("levels", [2, 50])
def test_tiny_grids(gpu_lib, oracle, ny, nx, levels):
    simplified(gpu_lib, oracle, tie_field(ny, nx, levels, ny * 100 + nx), 1.0, f"{nx}x{ny}")


@pytest.mark.parametrize("side", [24, 60, 90])
def test_heaps_up_to_and_past_the_shared_levels(gpu_lib, oracle, side):
    """White noise cancelled to the end: heaps from a few hundred entries to
    more than the 16,383 in shared memory, and lists of hundreds of runs."""
    f = np.random.default_rng(side).random((side, side), dtype=np.float32)
    st = simplified(gpu_lib, oracle, f, 0.35, f"noise {side}")
    assert st["cancels"] > side


@pytest.mark.parametrize("hubs", [3, 40, 300, 1500])
def test_long_neighbour_lists(gpu_lib, oracle, hubs):
    """One low basin with `hubs` separate shallow pits and as many peaks around
    it: the basin's lists hold about that many runs when they are merged."""
    rng = np.random.default_rng(hubs)
    n = max(12, int(4 * np.sqrt(hubs)) + 8)
    f = np.full((n, n), 0.5, np.float64) + rng.uniform(0, 1e-3, (n, n))
    at = rng.choice((n // 2 - 2) ** 2, hubs, replace=(n // 2 - 2) ** 2 < hubs)
    y, x = 2 * (at // (n // 2 - 2)) + 2, 2 * (at % (n // 2 - 2)) + 2
    f[y, x] = np.where(rng.random(hubs) < 0.5, 0.3, 0.7) + rng.uniform(-0.05, 0.05, hubs)
    f[1, 1] = -1.0
    simplified(gpu_lib, oracle, f.astype(np.float32), 0.02, f"{hubs} hubs")


@pytest.mark.parametrize("y,x,n", [(0, 0, 512), (512, 512, 512), (1024, 0, 400), (0, 2048, 400)])
def test_quantised_windows(gpu_lib, oracle, y, x, n):
    """Windows of the 4096x4096 quantised field: thousands of cancellations
    among lists whose lengths cross the line between short and long."""
    from mscomplex_gb300 import synth
    if not hasattr(test_quantised_windows, "field"):
        test_quantised_windows.field = synth.bumps4096q()
    f = np.ascontiguousarray(test_quantised_windows.field[y:y + n, x:x + n])
    simplified(gpu_lib, oracle, f, 0.01, f"window {y},{x} {n}")


@pytest.mark.parametrize("count", [152, 153, 330])
def test_batches_around_one_complex_per_sm(gpu_lib, oracle, count):
    """Up to 152 complexes take the launch shape of a single one, more take the
    one that shares SMs."""
    fields = [smooth_field(10 + i % 23, 12 + i % 17, i) if i % 3 else tie_field(8 + i % 19, 9 + i % 11, 6, i)
              for i in range(count)]
    fields[count // 2] = np.random.default_rng(7).random((70, 70), dtype=np.float32)
    b = gpu_lib.GridBatch().run(fields, 0.2)
    for i, f in enumerate(fields):
        r = full_rect(f)
        assert_same_complex(b.export(i), oracle.Dataset(f, r, r, tresh=0.2).msc(), f"grid {i}", keys=GRAPH)


@pytest.mark.parametrize("seed", range(3))
def test_infinite_heights(gpu_lib, oracle, seed):
    """An infinite range orders no key below another by more than equality:
    the pushes then take their plain order."""
    f = np.random.default_rng(seed).random((30, 34), dtype=np.float32)
    f[7, 9], f[23, 31] = np.inf, -np.inf
    simplified(gpu_lib, oracle, f, 0.1, f"infinite {seed}")
