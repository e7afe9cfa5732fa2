// chain_walk.h -- the walk along one chain of a saddle's disc, hop by hop
// (discs.cu), and the slots that describe the chain to the kernels after it.
// Without CUDA headers, so that it also compiles as plain C++.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CHAIN_HD __host__ __device__ __forceinline__
#else
#define CHAIN_HD inline
#endif

namespace dmsc {

constexpr uint32_t HOP_END = 0xFFFFFFFFu;
constexpr int SEG_LOG = 5, SEG_MAX = 1 << SEG_LOG;  // cells of a write piece: the jump pointer distance

enum : uint32_t {
  CHAIN_BRANCHES = 1,  // a hop without cells: a chain cell never branches
  CHAIN_CYCLE = 2,     // longer than the window has cells
  CHAIN_NO_SLOT = 4,
};

// The chain from ext-local edge e: its length, stored with its piece count as
// chain j of saddle s where that saddle's chains are kept.  C has the fields
// of ChainArgs that it names.  Every slot that is there is written: the sums
// over the slots and the kernels that index by them run before the host sees a
// fault.  A chain without an end is stored as one without cells and pieces.
template <class C>
CHAIN_HD unsigned long long chain_walk(const C &c, uint32_t s, uint32_t j, uint32_t e, uint32_t &fault) {
  unsigned long long L = 0;
  uint32_t nseg = 0;
  for (uint32_t x = e; x != HOP_END; x = c.hop_to[x]) {
    const uint32_t l = c.hop_len[x];
    if (l == 0) { fault |= CHAIN_BRANCHES; break; }
    L += l;
    nseg += (l + SEG_MAX - 1) / SEG_MAX;
    if (L > c.limit) {
      fault |= CHAIN_CYCLE;
      L = 0;
      e = HOP_END;
      break;
    }
  }
  if (!(c.big[s] & 1u)) {
    // piece slots: one per SEG_MAX cells of each hop, and one more for each level
    // where another of the saddle's chains ends inside this one (at most K - 1)
    if (j < c.cap) { c.cstart[j] = e; c.csaddle[j] = s; c.clen[j] = (uint32_t)L; c.cnseg[j] = L ? nseg + c.kc[s] - 1 : 0; }
    else fault |= CHAIN_NO_SLOT;
  }
  return L;
}

}  // namespace dmsc
