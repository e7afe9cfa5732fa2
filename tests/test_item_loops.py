"""CPU check, by reading the source, of the disc kernels' loops over the items
from cancelled extrema.  There may be up to 2^32 - 2 of them (lists are as long
as their 32-bit offsets reach), so near that many a 32-bit index wraps before
it passes the bound and the loop never ends; critical points stay below 2^30."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
THREADS, BLOCKS = 256, 152 * 16  # the largest launch of those kernels


def ends(bits, n):
    """Whether `for (i = last thread; i < n; i += threads)` ends with an index of so many bits."""
    i = THREADS * BLOCKS - 1
    i += (n - i) // (THREADS * BLOCKS) * (THREADS * BLOCKS)  # its last places
    for _ in range(3):
        if i >= n:
            return True
        i = (i + THREADS * BLOCKS) % (1 << bits)
    return False


@pytest.mark.parametrize("kernel,bound", [("k_seed_write", "n"), ("k_seed_chains", "sr.n"), ("k_seed_len", "sr.n"),
                                          ("k_seed_level0", "sr.n")])
def test_item_loops_end(kernel, bound):
    text = open(os.path.join(ROOT, "mscomplex_gb300", "csrc", "discs.cu")).read()
    body = text[text.index(f"void {kernel}("):]
    loop = re.search(r"for \((.+?) p = (.+?); p < ([\w.]+);", body)
    assert loop.group(3) == bound
    bits = {"uint32_t": 32, "unsigned long long": 64}[loop.group(1)]
    assert ends(bits, 2 ** 32 - 2)


def test_search_among_one_saddles_items():
    """Its middle is taken without the sum of both ends, which wraps beyond 2^31 items."""
    text = open(os.path.join(ROOT, "mscomplex_gb300", "csrc", "discs.cu")).read()
    body = text[text.index("uint32_t pushes_before("):]
    middle = re.search(r"const uint32_t m = (.+?);", body).group(1).replace("/", "//")
    lo, hi = 2 ** 32 - 9, 2 ** 32 - 3

    class U32(int):
        def __add__(self, o): return U32((int(self) + int(o)) % 2 ** 32)
        def __sub__(self, o): return U32((int(self) - int(o)) % 2 ** 32)
        def __floordiv__(self, o): return U32(int(self) // int(o))
        def __rshift__(self, o): return U32(int(self) >> int(o))

    assert lo <= eval(middle, {"lo": U32(lo), "hi": U32(hi)}) < hi
