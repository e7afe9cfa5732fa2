"""Cancellations multiply the counts of the asc / des multisets: lists of
thousands of equal entries, saddles with thousands of disc items, and fields
whose lists outgrow 32-bit offsets.  Noisy bumps at 5% of their range."""
import numpy as np
import pytest

from helpers import assert_same_complex, full_rect

pytestmark = pytest.mark.gpu

GRAPH = ("cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")


def noisy_bumps(n, seed):
    from mscomplex_gb300 import synth
    return synth.gaussian_bumps(n, n, 16, n / 32, n / 8, np.random.default_rng(seed), noise=1e-3)


def simplified(M, f, tresh=0.05):
    r = full_rect(f)
    ds = M.GridDataset(r, r).init(f).work()
    m = ds.writeout_connectivity()
    m.simplify_un_simplify(tresh)
    return ds, m


@pytest.mark.parametrize("n,seed", [(96, 12), (96, 20), (96, 4), (96, 10), (128, 19)])
def test_saddles_with_many_disc_items(gpu_lib, oracle, n, seed):
    """Up to 57, 132, 937, 4019 and 1180 items from cancelled extrema at one
    saddle: its chains around and past the 32 that are interleaved, and levels
    around and past a block's threads."""
    f = noisy_bumps(n, seed)
    r = full_rect(f)
    want = oracle.Dataset(f, r, r, tresh=0.05, fill_discs=True).msc()
    ds, m = simplified(gpu_lib, f)
    ds.post_merge_fill_discs(m)
    assert_same_complex(m.export(), want, f"{n} seed {seed}")


@pytest.mark.parametrize("seed", [231, 236, 391])
def test_lists_with_long_runs(gpu_lib, oracle, seed):
    """Runs of 13,770, 18,420 and 25,849 equal entries: one and two pieces of
    the list output."""
    f = noisy_bumps(256, seed)
    r = full_rect(f)
    _, m = simplified(gpu_lib, f)
    assert_same_complex(m.export(), oracle.Dataset(f, r, r, tresh=0.05).msc(), f"seed {seed}", keys=GRAPH)


def test_lists_beyond_their_offsets_are_refused(gpu_lib):
    """More than 2^32 - 1 entries: an error, and the complex as it was; in a
    batch that grid fails alone."""
    f = noisy_bumps(256, 207)
    r = full_rect(f)
    m = gpu_lib.GridDataset(r, r).init(f).work().writeout_connectivity()
    before = m.export()
    with pytest.raises(gpu_lib.DmscError, match="2\\^32"):
        m.simplify_un_simplify(0.05)
    assert_same_complex(m.export(), before, "after the refusal")
    g = noisy_bumps(96, 1)
    b = gpu_lib.GridBatch().run([g, f, g], 0.05, partial_ok=True)
    assert b.grid_status(1)[0] != 0 and "2^32" in b.grid_status(1)[1]
    _, alone = simplified(gpu_lib, g)
    for i in (0, 2):
        assert b.grid_status(i)[0] == 0
        assert_same_complex(b.export(i), alone.export(), f"grid {i}", keys=GRAPH)
