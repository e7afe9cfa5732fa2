"""Waits between warps that uncancel pairs side by side (csrc/warp_graph.cuh):
a wait during which no warp gets on ends with a status of its own, one for
another warp that is only slow does not end, and the long loops over a list
are seen as getting on.  A program of its own, with a short limit."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "warp_graph.cuh"
#include <cstdio>
#include <vector>
using namespace dmsc;

// Points 0 .. 7; asc(0) = {1, 2}, and 2 is cancelled with 3, whose asc list is
// {5 twice, 6}.  Uncancelling (0, 1) rewrites asc(0) from asc(3) once the list
// of the pair (3, 2), later on the cancellation list, is done.
struct Mem {
  uint32_t off[16], nrun[16], cap[16], total[16], pair_idx[8], ord[8], cellid[8];
  uint8_t flags[8];
  uint2 pool[64];
  uint32_t out[8];
};
enum { ALONE, SLOW, STOPPED };

__global__ void k_wait(Mem *m, int mode) {
  __shared__ TeamState team;
  __shared__ uint32_t done[2];
  if (threadIdx.x == 0) {
    team = TeamState{};
    team.top = 32;
    done[0] = done[1] = 0;
  }
  __syncthreads();
  WarpGraph W;
  W.G = Graph{8, m->cellid, m->flags, m->pair_idx, Lists{m->off, m->nrun, m->cap, m->total, m->pool, 32, 64}, nullptr, 0, ~0ull};
  W.lane = threadIdx.x & 31;
  W.stage = nullptr;
  W.nstage = 0;
  __shared__ uint2 stage[64];
  W.stage = stage;
  W.nstage = 64;
  W.team = &team;
  W.ord = m->ord;
  W.done = done;
  if (threadIdx.x < 32) {
    const bool ok = W.uncancel_list(0, 1, 0, 1);
    if (threadIdx.x == 0) {
      m->out[0] = ok;
      m->out[1] = W.G.fail;
      m->out[2] = team.late;
    }
  } else if (mode == SLOW) {  // gets on for many times the limit, then has the list done
    for (int i = 0; i < 2000; ++i) {
      __nanosleep(100000);
      if (W.lane == 0) W.moved_on();
      __syncwarp();
    }
    if (W.lane == 0) atomicOr(&done[0], 1u << (2 * (2 - 1) + 0));
  } else if (mode == STOPPED) {
    __nanosleep(1000);
    if (W.lane == 0) atomicExch(&team.fail, 1u);
  }
}

__global__ void k_long(uint2 *pool, uint2 *tmp, unsigned long long room, uint32_t n, uint32_t *desc, uint32_t *out) {
  __shared__ TeamState team;
  if (threadIdx.x == 0) {
    team = TeamState{};
    team.top = 0;
  }
  __syncwarp();
  WarpGraph W;
  W.G = Graph{1, nullptr, nullptr, nullptr, Lists{desc, desc + 2, desc + 4, desc + 6, pool, 0, 2ull * n + 64}, tmp, room, ~0ull};
  W.lane = threadIdx.x;
  W.stage = nullptr;
  W.nstage = 0;
  W.team = &team;
  for (uint32_t i = W.lane; i < n; i += 32) tmp[i] = make_uint2((i * 2654435761u) % 977u, 1u);
  __syncwarp();
  const bool ok = W.set_list(0, tmp, n);
  if (W.lane == 0) {
    out[0] = ok && !W.G.fail;
    out[1] = team.beat;
    out[2] = desc[2];
    out[3] = desc[6];
  }
}

static int fails = 0;
static void expect(bool ok, const char *what) { if (!ok) { std::printf("FAIL %s\n", what); ++fails; } }
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { std::printf("%s: %s\n", #x, cudaGetErrorString(e_)); return 2; } } while (0)

int main() {
  Mem *d = nullptr, h0{}, h;
  for (int l = 0; l < 16; ++l) { h0.off[l] = 2 * l; h0.cap[l] = 2; }
  auto list = [&](uint32_t l, std::vector<uint2> v) {
    h0.nrun[l] = (uint32_t)v.size();
    for (size_t i = 0; i < v.size(); ++i) { h0.pool[h0.off[l] + i] = v[i]; h0.total[l] += v[i].y; }
  };
  list(0, {make_uint2(1, 1), make_uint2(2, 1)});
  list(6, {make_uint2(5, 2), make_uint2(6, 1)});
  h0.flags[0] = h0.flags[1] = h0.flags[2] = h0.flags[3] = F_CANCELLED | F_BCANCEL;
  h0.pair_idx[0] = 1; h0.pair_idx[1] = 0; h0.pair_idx[2] = 3; h0.pair_idx[3] = 2;
  h0.ord[0] = h0.ord[1] = 1; h0.ord[2] = h0.ord[3] = 2;
  CK(cudaMalloc(&d, sizeof(Mem)));
  for (int mode : {ALONE, SLOW, STOPPED}) {
    CK(cudaMemcpy(d, &h0, sizeof(Mem), cudaMemcpyHostToDevice));
    k_wait<<<1, 64>>>(d, mode);
    CK(cudaDeviceSynchronize());
    CK(cudaMemcpy(&h, d, sizeof(Mem), cudaMemcpyDeviceToHost));
    std::printf("mode %d: ok %u fail %u late %u, asc(0) %u runs\n", mode, h.out[0], h.out[1], h.out[2], h.nrun[0]);
    if (mode == ALONE) expect(h.out[0] == 1 && h.out[1] == 1 && h.out[2] == 1, "a wait that nobody ends has its own status");
    if (mode == STOPPED) expect(h.out[0] == 1 && h.out[1] == 1 && h.out[2] == 0, "a stopped wait is no wait that ran out");
    if (mode == SLOW) {
      expect(h.out[0] == 1 && h.out[1] == 0 && h.out[2] == 0, "a slow warp is waited for");
      const uint2 *p = h.pool + h.off[0];
      expect(h.nrun[0] == 2 && h.total[0] == 3 && p[0].x == 5 && p[0].y == 2 && p[1].x == 6 && p[1].y == 1, "its list is used");
    }
  }
  const uint32_t n = 20000;
  uint2 *buf = nullptr;
  uint32_t *desc = nullptr, o[4];
  CK(cudaMalloc(&buf, sizeof(uint2) * (32768 + 2 * n + 64)));
  CK(cudaMalloc(&desc, sizeof(uint32_t) * 16));
  for (unsigned long long room : {32768ull, (unsigned long long)n}) {  // sorted by the warp, and by one lane
    CK(cudaMemset(desc, 0, sizeof(uint32_t) * 16));
    k_long<<<1, 32>>>(buf + 32768, buf, room, n, desc, desc + 8);
    CK(cudaDeviceSynchronize());
    CK(cudaMemcpy(o, desc + 8, sizeof o, cudaMemcpyDeviceToHost));
    std::printf("room %llu: ok %u beats %u runs %u total %u\n", room, o[0], o[1], o[2], o[3]);
    expect(o[0] == 1 && o[2] == 977 && o[3] == n, "a long list");
    expect(o[1] >= 10, "its loops are seen to get on");
  }
  return fails != 0;
}
"""


def test_waits_of_a_team(gpu_lib, tmp_path):
    from mscomplex_gb300 import build as B
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, "-DDMSC_WAIT_POLLS=(1ull<<16)", str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
