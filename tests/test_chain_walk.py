"""CPU check of the walk along a disc's chain (csrc/chain_walk.h, compiled as
plain C++): the slots of every chain are written, also of one that never ends,
whose walk stops at the limit.  The sums over the slots and the kernels that
index by them run before the host reads the status, so a slot left as it was
would be memory of another call."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "chain_walk.h"
#include <cstdio>
using namespace dmsc;

struct Args {
  const uint32_t *hop_to;
  const uint16_t *hop_len;
  uint32_t *kc;
  uint8_t *big;
  uint32_t *cstart, *csaddle, *clen, *cnseg;
  uint32_t cap;
  unsigned long long limit;
};
static int fails = 0;
static void expect(bool ok, const char *what) { if (!ok) { std::printf("FAIL %s\n", what); ++fails; } }

int main() {
  // hops 0 -> 1 -> end; 2 -> 3 -> 2 without end; 4: no cells
  const uint32_t to[5] = {1, HOP_END, 3, 2, HOP_END};
  const uint16_t len[5] = {40, 33, 7, 9, 0};
  uint32_t kc[1] = {3}, slot[4][4];
  uint8_t big[1] = {0};
  for (auto &a : slot) for (uint32_t &v : a) v = 0xA5A5A5A5u;  // another call's
  const Args c{to, len, kc, big, slot[0], slot[1], slot[2], slot[3], 3, 1000};
  auto is = [&](uint32_t j, uint32_t e, uint32_t l, uint32_t n) {
    return slot[0][j] == e && slot[1][j] == 0 && slot[2][j] == l && slot[3][j] == n;
  };
  uint32_t fault = 0;
  expect(chain_walk(c, 0, 0, 0, fault) == 73 && fault == 0, "an ordinary chain");
  expect(is(0, 0, 73, 2 + 2 + 2), "its slots");
  expect(chain_walk(c, 0, 1, 2, fault) == 0 && fault == CHAIN_CYCLE, "a chain without end");
  expect(is(1, HOP_END, 0, 0), "it is stored without cells and pieces");
  fault = 0;
  expect(chain_walk(c, 0, 2, 4, fault) == 0 && fault == CHAIN_BRANCHES, "a hop without cells");
  expect(slot[0][2] != 0xA5A5A5A5u && slot[1][2] == 0 && slot[2][2] == 0 && slot[3][2] <= 2, "its slots");
  fault = 0;
  chain_walk(c, 0, 3, 0, fault);
  expect(fault == CHAIN_NO_SLOT && slot[0][3] == 0xA5A5A5A5u, "no slot past the capacity");
  fault = 0;
  big[0] = 1;  // this saddle's chains are not kept
  expect(chain_walk(c, 0, 0, 2, fault) == 0 && fault == CHAIN_CYCLE && is(0, 0, 73, 6), "a saddle with many chains");
  return fails != 0;
}
"""


def test_every_chain_slot_is_written(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "mscomplex_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
