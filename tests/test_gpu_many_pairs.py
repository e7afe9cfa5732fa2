"""Uncancelling more pairs than shared memory tracks (65,536): the bits of the
lists that are done then lie in global memory.  Compared with the oracle's."""
import numpy as np
import pytest

from helpers import assert_same_complex, full_rect

pytestmark = pytest.mark.gpu

GRAPH = ("cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")


def test_more_pairs_than_shared_memory_tracks(gpu_lib, oracle):
    f = np.random.default_rng(800).random((800, 800), dtype=np.float32)
    r = full_rect(f)
    want = oracle.Dataset(f, r, r, tresh=0.03).msc()
    m = gpu_lib.GridDataset(r, r).init(f).work().writeout_connectivity()
    st = m.simplify_un_simplify(0.03)
    assert st["cancels"] > 65536
    assert_same_complex(m.export(), want, "noise 800", keys=GRAPH)
