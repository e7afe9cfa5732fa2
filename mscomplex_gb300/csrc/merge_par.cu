// merge_par.cu -- the piece merges of one tree level with the bulk of their
// work spread over the GPU: GridMSComplex::merge_up and merge_down
// (dmsc/src/grid_mscomplex.cpp:24-322) for complexes of millions of critical
// points, where one thread per merge (merge.cu) would walk every critical
// point and every arc in sequence.
//
// merge_up (:24-156) splits into
//   * the union of the critical points (:56-75): A's uncancelled points keep
//     their order, then B's uncancelled points whose cell A does not hold --
//     a scan over each input gives every point its index in the result;
//   * the boundary pairs (:84-92): each input's uncancelled boundary-cancelable
//     point takes its partner's index (B's assignment after A's, as the
//     reference's loop order leaves it);
//   * the connectivity (:77-122): the result's list of a point is the
//     multiset union of A's list and B's list (B's without arcs inside the
//     shared boundary when the point itself lies on it), restricted to
//     uncancelled points -- counts, a scan, a scatter, and a sort of each list
//     by index (the ascending order in which a std::multiset iterates);
//   * the cancellations along the shared boundary (:124-153), row-major and
//     order dependent among cells that touch a common point: on the mutable
//     graph, one block per group of such cells (k_merge_up_seq), all merges of
//     the level in one launch.
// merge_down (:158-322) splits into
//   * the uncancellations along the shared boundary (:172-201): one block per
//     parent (k_merge_down_seq), all merges of the level in one launch;
//   * the parent's boundary-cancelable points pushed into each child
//     (:207-281): the points it adds to the child are numbered by a scan over
//     the sequence of additions the reference's loop makes (down_child);
//   * every child point whose cell the parent holds takes the parent's
//     lists, restricted to points the child holds (:283-320): counts, a scan,
//     a scatter and a sort per list into the child's new CSR arrays.
// A step whose outcome only the one-thread restatement reproduces (a partner
// missing from the union, where the reference's std::map::operator[] would
// insert index 0; a boundary-cancelable point whose partner does not point
// back) reports ST_FALLBACK and the caller reruns the level with the
// one-thread merges.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <string>
#include <vector>

#include "dmsc_common.cuh"
#include "dmsc_internal.h"
#include "grid_types.h"
#include "host_pool.h"
#include "merge_graph.cuh"
#include "smem_limit.h"
#include "warp_graph.cuh"

namespace dmsc {

namespace {

unsigned nblk(long long n) {
  long long b = (n + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  return (unsigned)(b < 1 ? 1 : b);
}

#define GRID_LOOP(i, n) for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)(n); i += (long long)gridDim.x * blockDim.x)

// Cell id -> critical-point index over a box of cell coordinates (the same
// table a merged graph keeps).  Entries are written and read in separate
// launches; each cell is written once.
struct CellTab {
  uint32_t *tab;
  int x0, y0, w, h;
  __device__ long long slot(uint32_t cid) const {
    const int x = (int)(cid & 0xffffu) - x0, y = (int)(cid >> 16) - y0;
    if (x < 0 || y < 0 || x >= w || y >= h) return -1;
    return (long long)y * w + x;
  }
  __device__ uint32_t find(uint32_t cid) const {
    const long long s = slot(cid);
    return s < 0 ? NO_CP : tab[s];
  }
  __device__ bool insert(uint32_t cid, uint32_t v) {
    const long long s = slot(cid);
    if (s < 0) return false;
    tab[s] = v;
    return true;
  }
};

__device__ __forceinline__ bool cancelled(const uint8_t *fl, uint32_t i) { return fl[i] & F_CANCELLED; }

// ---------------------------------------------------------------------------
// sorting every list of a CSR array by value
// ---------------------------------------------------------------------------
constexpr uint32_t SS_THREAD = 32, SS_BLOCK = 8192;

// Segments of up to SS_THREAD values: insertion sort by one thread; longer
// ones are queued (up to SS_BLOCK for one block each, beyond for the radix
// sort).  `need` (may be null) marks the segments that can be out of order.
__global__ void k_ss_small(long long nseg, const uint32_t *__restrict__ off, const uint8_t *__restrict__ need,
                           uint32_t *__restrict__ vals, uint32_t *__restrict__ q_block, uint32_t *__restrict__ n_block,
                           uint32_t *__restrict__ q_huge, uint32_t *__restrict__ n_huge) {
  GRID_LOOP(s, nseg) {
    if (need && !need[s]) continue;
    const uint32_t b = off[s], n = off[s + 1] - b;
    if (n <= 1) continue;
    if (n > SS_THREAD) {
      if (n > SS_BLOCK) q_huge[atomicAdd(n_huge, 1u)] = (uint32_t)s;
      else q_block[atomicAdd(n_block, 1u)] = (uint32_t)s;
      continue;
    }
    uint32_t v[SS_THREAD];
    for (uint32_t i = 0; i < n; ++i) v[i] = vals[b + i];
    for (uint32_t i = 1; i < n; ++i) {
      const uint32_t x = v[i];
      uint32_t j = i;
      while (j > 0 && v[j - 1] > x) { v[j] = v[j - 1]; --j; }
      v[j] = x;
    }
    for (uint32_t i = 0; i < n; ++i) vals[b + i] = v[i];
  }
}

// queued segments of up to SS_BLOCK values: one block each, bitonic sort in shared memory
__global__ void __launch_bounds__(512) k_ss_block(const uint32_t *__restrict__ off, uint32_t *__restrict__ vals,
                                                  const uint32_t *__restrict__ q, const uint32_t *__restrict__ nq) {
  __shared__ uint32_t sh[SS_BLOCK];
  const uint32_t count = *nq;
  for (uint32_t k = blockIdx.x; k < count; k += gridDim.x) {
    const uint32_t s = q[k], b = off[s], n = off[s + 1] - b;
    if (n <= 1024) {  // rank sort: each value's place is the count of values before it
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) sh[i] = vals[b + i];
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t v = sh[i];
        uint32_t r = 0;
        for (uint32_t j = 0; j < n; ++j) {
          const uint32_t u = sh[j];
          r += (u < v) || (u == v && j < i);
        }
        vals[b + r] = v;
      }
      __syncthreads();
      continue;
    }
    uint32_t p2 = 1;
    while (p2 < n) p2 <<= 1;
    for (uint32_t i = threadIdx.x; i < p2; i += blockDim.x) sh[i] = i < n ? vals[b + i] : 0xFFFFFFFFu;
    __syncthreads();
    for (uint32_t size = 2; size <= p2; size <<= 1)
      for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
        for (uint32_t i = threadIdx.x; i < p2; i += blockDim.x) {
          const uint32_t j = i ^ stride;
          if (j > i) {
            const bool up = (i & size) == 0;
            const uint32_t x = sh[i], y = sh[j];
            if ((x > y) == up) { sh[i] = y; sh[j] = x; }
          }
        }
        __syncthreads();
      }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) vals[b + i] = sh[i];
    __syncthreads();
  }
}

// Sorts segments [off[s], off[s+1]) of vals for s < nseg where need[s] (all
// when need is null).  `off` is on the device; synchronises `st` once.
cudaError_t sort_segments(long long nseg, const uint32_t *off, uint32_t *vals, const uint8_t *need, cudaStream_t st) {
  if (nseg <= 0) return cudaSuccess;
  uint32_t *buf = nullptr;
  cudaError_t e = cudaMallocAsync((void **)&buf, 4ull * (2 * nseg + 4), st);
  if (e != cudaSuccess) return e;
  uint32_t *q_block = buf, *q_huge = buf + nseg, *cnt = buf + 2 * nseg;
  e = cudaMemsetAsync(cnt, 0, 16, st);
  if (e == cudaSuccess) {
    k_ss_small<<<nblk(nseg), 256, 0, st>>>(nseg, off, need, vals, q_block, cnt, q_huge, cnt + 1);
    k_ss_block<<<152 * 2, 512, 0, st>>>(off, vals, q_block, cnt);
    DMSC_LAUNCHED(2);
    e = cudaGetLastError();
  }
  uint32_t nh = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&nh, cnt + 1, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && nh) {  // rare: lists longer than SS_BLOCK, one radix sort each
    std::vector<uint32_t> segs(nh), o0(nh), o1(nh);
    e = cudaMemcpy(segs.data(), q_huge, 4ull * nh, cudaMemcpyDeviceToHost);
    for (uint32_t k = 0; k < nh && e == cudaSuccess; ++k) {
      e = cudaMemcpy(&o0[k], off + segs[k], 4, cudaMemcpyDeviceToHost);
      if (e == cudaSuccess) e = cudaMemcpy(&o1[k], off + segs[k] + 1, 4, cudaMemcpyDeviceToHost);
    }
    for (uint32_t k = 0; k < nh && e == cudaSuccess; ++k) {
      const long long n = (long long)o1[k] - o0[k];
      uint32_t *tmp = nullptr;
      e = cudaMallocAsync((void **)&tmp, 12ull * n, st);
      if (e != cudaSuccess) break;
      e = cudaMemsetAsync(tmp, 0, 4ull * n, st);
      if (e == cudaSuccess) e = radix_sort_pairs(vals + o0[k], tmp, tmp + n, tmp + 2 * n, n, 32, st);
      cudaFreeAsync(tmp, st);
    }
  }
  cudaFreeAsync(buf, st);
  return e;
}

// ---------------------------------------------------------------------------
// merge_up: union, boundary pairs, connectivity
// ---------------------------------------------------------------------------
struct CsrIn {  // a complex being read (device arrays)
  long long n;
  const uint32_t *cellid, *pair, *aoff, *asc, *doff, *des;
  const float *fn;
  const uint8_t *flags;
};
struct CsrOut {
  uint32_t *cellid, *pair, *aoff, *asc, *doff, *des;
  float *fn;
  uint8_t *flags;
};

CsrIn csr_in(const dmsc_msc &m) {
  return CsrIn{m.ncp, m.cellid.p, m.pair_idx.p, m.aoff.p, m.asc.p, m.doff.p, m.des.p, m.fn.p, m.flags.p};
}

__global__ void k_keep(CsrIn a, uint32_t *keep) {
  GRID_LOOP(j, a.n) keep[j] = cancelled(a.flags, (uint32_t)j) ? 0u : 1u;
}

// shallow_replicate_cp (grid_mscomplex.cpp:7-22): flags copied, partner unset
__device__ __forceinline__ void put_cp(const CsrIn &a, long long j, uint32_t d, CsrOut &o) {
  o.cellid[d] = a.cellid[j];
  o.fn[d] = a.fn[j];
  o.flags[d] = a.flags[j] & (F_CANCELLED | F_STRANG | F_BCANCEL);
  o.pair[d] = NO_CP;
}

// A's uncancelled points: index = scan of the keep flags
__global__ void k_up_a(CsrIn a, const uint32_t *idx, CellTab H, CsrOut o, uint32_t *status) {
  GRID_LOOP(j, a.n) {
    if (cancelled(a.flags, (uint32_t)j)) continue;
    if (!H.insert(a.cellid[j], idx[j])) { atomicOr(status, ST_SIMPLIFY_LIMIT); continue; }
    put_cp(a, j, idx[j], o);
  }
}

// B's uncancelled points: the index of A's copy, or new (counted by isnew)
__global__ void k_up_b_classify(CsrIn b, CellTab H, uint32_t *idx, uint32_t *isnew) {
  GRID_LOOP(j, b.n) {
    uint32_t d = NO_CP, nw = 0;
    if (!cancelled(b.flags, (uint32_t)j)) {
      d = H.find(b.cellid[j]);
      nw = d == NO_CP;
    }
    idx[j] = d;
    isnew[j] = nw;
  }
}

__global__ void k_up_b_new(CsrIn b, const uint32_t *isnew, const uint32_t *pos, const uint32_t *na, CellTab H, uint32_t *idx,
                           CsrOut o, uint32_t *status) {
  const uint32_t base = *na;
  GRID_LOOP(j, b.n) {
    if (!isnew[j]) continue;
    const uint32_t d = base + pos[j];
    idx[j] = d;
    if (!H.insert(b.cellid[j], d)) { atomicOr(status, ST_SIMPLIFY_LIMIT); continue; }
    put_cp(b, j, d, o);
  }
}

// boundary pairs (:84-92) of one input; idx = the result index of each point
__global__ void k_up_pairs(CsrIn a, const uint32_t *idx, CellTab H, uint32_t *opair, uint32_t *status) {
  GRID_LOOP(j, a.n) {
    const uint8_t fl = a.flags[j];
    if ((fl & F_CANCELLED) || !(fl & F_BCANCEL)) continue;
    const uint32_t p = a.pair[j];
    if (p >= (uint32_t)a.n) { atomicOr(status, ST_INVARIANT); continue; }
    const uint32_t t = H.find(a.cellid[p]);
    if (t == NO_CP) { atomicOr(status, ST_FALLBACK); continue; }
    opair[idx[j]] = t;
  }
}

// list lengths: A's stored, B's added (each result point has at most one
// source point in each input); mix marks the lists that B contributed to
__global__ void k_up_count(CsrIn a, const uint32_t *idx, bool second, CRect ixn, uint32_t *tot_a, uint32_t *tot_d,
                           uint8_t *mix, uint32_t *status) {
  GRID_LOOP(j, a.n) {
    if (cancelled(a.flags, (uint32_t)j)) continue;
    const uint32_t d = idx[j], cid = a.cellid[j];
    const bool cmn = second && ixn.contains(px_(cid), py_(cid));
    uint32_t c[2] = {0, 0};
    for (int w = 0; w < 2; ++w) {
      const uint32_t *o = w ? a.doff : a.aoff, *l = w ? a.des : a.asc;
      for (uint32_t q = o[j]; q < o[j + 1]; ++q) {
        const uint32_t r = l[q];
        if (r >= (uint32_t)a.n) { atomicOr(status, ST_INVARIANT); continue; }
        if (cancelled(a.flags, r)) continue;
        if (cmn && ixn.contains(px_(a.cellid[r]), py_(a.cellid[r]))) continue;
        ++c[w];
      }
    }
    if (second) {
      tot_a[d] += c[0];
      tot_d[d] += c[1];
      if (c[0] + c[1]) mix[d] = 1;
    } else {
      tot_a[d] = c[0];
      tot_d[d] = c[1];
    }
  }
}

// entries: A's from the front of each list (in order), B's from the back
__global__ void k_up_write(CsrIn a, const uint32_t *idx, bool second, CRect ixn, CsrOut o) {
  GRID_LOOP(j, a.n) {
    if (cancelled(a.flags, (uint32_t)j)) continue;
    const uint32_t d = idx[j], cid = a.cellid[j];
    const bool cmn = second && ixn.contains(px_(cid), py_(cid));
    for (int w = 0; w < 2; ++w) {
      const uint32_t *io = w ? a.doff : a.aoff, *l = w ? a.des : a.asc;
      uint32_t *oo = w ? o.doff : o.aoff, *ol = w ? o.des : o.asc;
      const uint32_t lo = oo[d], hi = oo[d + 1];
      uint32_t p = second ? hi : lo;
      for (uint32_t q = io[j]; q < io[j + 1]; ++q) {
        const uint32_t r = l[q];
        if (r >= (uint32_t)a.n || cancelled(a.flags, r)) continue;
        if (cmn && ixn.contains(px_(a.cellid[r]), py_(a.cellid[r]))) continue;
        if (second) { if (p > lo) ol[--p] = idx[r]; }
        else if (p < hi) ol[p++] = idx[r];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// merge_down: parent checks, its boundary-cancelable list, the child rewrite
// ---------------------------------------------------------------------------
// "all cps ought to be uncancelled" (:209) and the boundary-cancelable flags
__global__ void k_down_check(MGraph P, uint32_t *bflag, uint32_t *status) {
  GRID_LOOP(j, P.G.ncp) {
    const uint8_t fl = P.G.flags[j];
    if (fl & F_CANCELLED) atomicOr(status, ST_INVARIANT);
    bflag[j] = (fl & F_BCANCEL) ? 1u : 0u;
  }
}

// the boundary-cancelable points in index order, a bound on the points they
// can add to a child (themselves, their partners, their list entries) and
// the box of those points' cells (box: l, b, r, t)
__device__ __forceinline__ void box_add(int b[4], uint32_t cid) {
  const int x = (int)(cid & 0xffffu), y = (int)(cid >> 16);
  b[0] = min(b[0], x); b[1] = min(b[1], y); b[2] = max(b[2], x); b[3] = max(b[3], y);
}
__global__ void k_down_list(MGraph P, const uint32_t *bflag, const uint32_t *pos, uint32_t *jb,
                            unsigned long long *adds, int *box) {
  unsigned long long mine = 0;
  int b[4] = {1 << 30, 1 << 30, -1, -1};
  GRID_LOOP(j, P.G.ncp) {
    if (!bflag[j]) continue;
    jb[pos[j]] = (uint32_t)j;
    mine += 2ull + P.G.L.nrun[2 * j] + P.G.L.nrun[2 * j + 1];
    box_add(b, P.G.cellid[j]);
    const uint32_t sp = P.G.pair_idx[j];
    if (sp < P.G.ncp) box_add(b, P.G.cellid[sp]);
    for (int w = 0; w < 2; ++w) {
      const uint2 *r = P.G.runs(2 * j + w);
      for (uint32_t q = 0; q < P.G.L.nrun[2 * j + w]; ++q)
        if (r[q].x < P.G.ncp) box_add(b, P.G.cellid[r[q].x]);
    }
  }
  if (mine) atomicAdd(adds, mine);
  if (b[2] >= 0) {
    atomicMin(box, b[0]); atomicMin(box + 1, b[1]); atomicMax(box + 2, b[2]); atomicMax(box + 3, b[3]);
  }
}

// ---------------------------------------------------------------------------
// merge_down into one child (:207-320) without a mutable graph of the child.
// The parent's boundary-cancelable points j (in index order, the list jb)
// come in pairs (j, sp).  A pair whose two cells the child lacks is skipped;
// when it holds exactly one, the first of the pair (lower index) adds the
// other; the pair is then marked boundary-cancelable and paired in the child
// unless both cells were already there with the mark.  The first of each
// non-skipped point's list entries that the child lacks adds it, in the
// order the reference's loop meets them: so every addition is an event in
// one sequence (per point: its partner, then its asc, then its des entries),
// and a scan over that sequence numbers the added points.  Finally every
// child point whose cell the parent holds takes the parent's lists,
// restricted to the points the child holds (for boundary-cancelable points
// the child holds them all by then); the others keep their own.
// ---------------------------------------------------------------------------
enum : uint8_t { DC_SKIP = 1, DC_ADD = 2, DC_FIRST = 4, DC_S0 = 8, DC_P0 = 16 };

struct DcArgs {
  MGraph P;                 // the parent after its boundary uncancellations
  const uint32_t *jb;       // its boundary-cancelable points, ascending
  uint32_t njb;
  CsrIn c;                  // the child before the merge
  CellTab tab;              // child cell -> index (initial points, then the added ones)
  CellTab first;            // missing cell -> position of its first list event
  uint32_t *cnt, *base, *addsrc;
  uint8_t *kind;            // per boundary point
  uint32_t *addf, *rank;    // per event
  CsrOut o;                 // the child's point arrays after the merge
  uint32_t ncp0;
  uint32_t *status;
};

__global__ void k_dc_table(CsrIn c, CellTab tab, uint32_t *status) {
  GRID_LOOP(i, c.n) {
    if (!tab.insert(c.cellid[i], (uint32_t)i)) atomicOr(status, ST_INVARIANT);
  }
}

__global__ void k_dc_classify(DcArgs a) {
  GRID_LOOP(q, a.njb) {
    const uint32_t j = a.jb[q], sp = a.P.G.pair_idx[j];
    uint8_t kd = 0;
    uint32_t n = 0;
    if (sp >= a.P.G.ncp || sp == j || a.P.G.pair_idx[sp] != j || !(a.P.G.flags[sp] & F_BCANCEL)) {
      atomicOr(a.status, ST_FALLBACK);  // not a plain pair: the one-thread merge handles it
      kd = DC_SKIP;
    } else {
      const bool s0 = a.tab.find(a.P.G.cellid[j]) != NO_CP, p0 = a.tab.find(a.P.G.cellid[sp]) != NO_CP;
      if (s0) kd |= DC_S0;
      if (p0) kd |= DC_P0;
      if (j < sp) kd |= DC_FIRST;
      if (!s0 && !p0) kd |= DC_SKIP;
      else {
        if (j < sp && s0 != p0) { kd |= DC_ADD; a.addsrc[q] = s0 ? sp : j; ++n; }
        n += a.P.G.L.nrun[2 * j] + a.P.G.L.nrun[2 * j + 1];
      }
    }
    a.kind[q] = kd;
    a.cnt[q] = n;
  }
}

// the first list event of every cell the child lacks
__global__ void k_dc_first(DcArgs a) {
  GRID_LOOP(q, a.njb) {
    const uint8_t kd = a.kind[q];
    if (kd & DC_SKIP) continue;
    const uint32_t j = a.jb[q];
    uint32_t pos = a.base[q] + ((kd & DC_ADD) ? 1 : 0);
    for (int w = 0; w < 2; ++w) {
      const uint2 *r = a.P.G.runs(2 * j + w);
      for (uint32_t k = 0; k < a.P.G.L.nrun[2 * j + w]; ++k, ++pos) {
        const uint32_t x = r[k].x;
        if (x >= a.P.G.ncp || (a.P.G.flags[x] & F_BCANCEL)) { atomicOr(a.status, ST_INVARIANT); continue; }
        const uint32_t cc = a.P.G.cellid[x];
        if (a.tab.find(cc) != NO_CP) continue;
        const long long sl = a.first.slot(cc);
        if (sl < 0) atomicOr(a.status, ST_INVARIANT);
        else atomicMin(a.first.tab + sl, pos);
      }
    }
  }
}

__global__ void k_dc_addflags(DcArgs a) {
  GRID_LOOP(q, a.njb) {
    const uint8_t kd = a.kind[q];
    if (kd & DC_SKIP) continue;
    const uint32_t j = a.jb[q];
    uint32_t pos = a.base[q];
    if (kd & DC_ADD) a.addf[pos++] = 1;
    for (int w = 0; w < 2; ++w) {
      const uint2 *r = a.P.G.runs(2 * j + w);
      for (uint32_t k = 0; k < a.P.G.L.nrun[2 * j + w]; ++k, ++pos) {
        const uint32_t x = r[k].x;
        if (x >= a.P.G.ncp) continue;
        const uint32_t cc = a.P.G.cellid[x];
        const long long sl = a.first.slot(cc);
        a.addf[pos] = (a.tab.find(cc) == NO_CP && sl >= 0 && a.first.tab[sl] == pos) ? 1u : 0u;
      }
    }
  }
}

// shallow_replicate_cp of parent point x as child point d
__device__ __forceinline__ void dc_put(DcArgs &a, uint32_t x, uint32_t d) {
  const uint32_t cid = a.P.G.cellid[x];
  a.o.cellid[d] = cid;
  a.o.fn[d] = a.P.fn[x];
  a.o.flags[d] = a.P.G.flags[x] & (F_CANCELLED | F_STRANG | F_BCANCEL);
  a.o.pair[d] = NO_CP;
  if (!a.tab.insert(cid, d)) atomicOr(a.status, ST_INVARIANT);
}

__global__ void k_dc_add(DcArgs a) {
  GRID_LOOP(q, a.njb) {
    const uint8_t kd = a.kind[q];
    if (kd & DC_SKIP) continue;
    const uint32_t j = a.jb[q];
    uint32_t pos = a.base[q];
    if (kd & DC_ADD) { dc_put(a, a.addsrc[q], a.ncp0 + a.rank[pos]); ++pos; }
    for (int w = 0; w < 2; ++w) {
      const uint2 *r = a.P.G.runs(2 * j + w);
      for (uint32_t k = 0; k < a.P.G.L.nrun[2 * j + w]; ++k, ++pos)
        if (a.addf[pos]) dc_put(a, r[k].x, a.ncp0 + a.rank[pos]);
    }
  }
}

// the pairing of each non-skipped pair, once (by its first point)
__global__ void k_dc_pairing(DcArgs a) {
  GRID_LOOP(q, a.njb) {
    const uint8_t kd = a.kind[q];
    if ((kd & DC_SKIP) || !(kd & DC_FIRST)) continue;
    const uint32_t j = a.jb[q], sp = a.P.G.pair_idx[j];
    const uint32_t d1 = a.tab.find(a.P.G.cellid[j]), d2 = a.tab.find(a.P.G.cellid[sp]);
    if (d1 == NO_CP || d2 == NO_CP) { atomicOr(a.status, ST_INVARIANT); continue; }
    const bool set = (kd & DC_ADD) || !(a.o.flags[d1] & F_BCANCEL) || !(a.o.flags[d2] & F_BCANCEL);
    if (!set) continue;
    a.o.flags[d1] |= F_BCANCEL;
    a.o.flags[d2] |= F_BCANCEL;
    a.o.pair[d1] = d2;
    a.o.pair[d2] = d1;
  }
}

// the parent point (if any) whose lists each child point takes
__global__ void k_dc_src(DcArgs a, uint32_t n, uint32_t *src) {
  GRID_LOOP(d, n) src[d] = a.P.find(a.o.cellid[d]);
}

__global__ void k_dc_count(DcArgs a, uint32_t n, const uint32_t *src, uint32_t *tot_a, uint32_t *tot_d, uint8_t *need) {
  GRID_LOOP(d, n) {
    const uint32_t j = src[d];
    for (int w = 0; w < 2; ++w) {
      uint32_t c = 0;
      if (j == NO_CP) {
        const uint32_t *off = w ? a.c.doff : a.c.aoff;
        if (d < a.ncp0) c = off[d + 1] - off[d];
      } else {
        const uint2 *r = a.P.G.runs(2 * j + w);
        for (uint32_t k = 0; k < a.P.G.L.nrun[2 * j + w]; ++k)
          if (r[k].x < a.P.G.ncp && a.tab.find(a.P.G.cellid[r[k].x]) != NO_CP) c += r[k].y;
      }
      (w ? tot_d : tot_a)[d] = c;
    }
    need[d] = j != NO_CP;
  }
}

__global__ void k_dc_write(DcArgs a, uint32_t n, const uint32_t *src) {
  GRID_LOOP(d, n) {
    const uint32_t j = src[d];
    for (int w = 0; w < 2; ++w) {
      const uint32_t *oo = w ? a.o.doff : a.o.aoff;
      uint32_t p = oo[d];
      const uint32_t end = oo[d + 1];
      uint32_t *ol = w ? a.o.des : a.o.asc;
      if (j == NO_CP) {
        if (d >= a.ncp0) continue;
        const uint32_t *off = w ? a.c.doff : a.c.aoff, *l = w ? a.c.des : a.c.asc;
        for (uint32_t q = off[d]; q < off[d + 1] && p < end; ++q) ol[p++] = l[q];
      } else {
        const uint2 *r = a.P.G.runs(2 * j + w);
        for (uint32_t k = 0; k < a.P.G.L.nrun[2 * j + w]; ++k) {
          if (r[k].x >= a.P.G.ncp) continue;
          const uint32_t ci = a.tab.find(a.P.G.cellid[r[k].x]);
          if (ci == NO_CP) continue;
          for (uint32_t c = 0; c < r[k].y && p < end; ++c) ol[p++] = ci;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// the boundary steps of a level, all jobs in one launch: merge_up up to
// UP_BLOCKS blocks per job (one where its cells go in plain order), merge_down
// one block per job
// ---------------------------------------------------------------------------
enum SeqKind : int { SEQ_UP_CANCEL = 0, SEQ_DOWN_BOUNDARY = 1 };
struct SeqJob {
  int kind, g0;
  CRect ixn;
  int win = 0, min_commits = 0;  // SEQ_UP_CANCEL: rounds window (0: groups of cells) and hand-off rate
};

// Loads, across the GPU, what the boundary step of a job will read -- the
// boundary points, their partners, their lists and their neighbours' list
// descriptors -- so that the step finds it in L2 instead of DRAM.  Reads
// only; the sum is stored only under a condition that never holds, so the
// loads are kept.
__device__ __forceinline__ uint32_t touch_cp(const MGraph &M, uint32_t c) {
  if (c >= M.G.ncp) return 0;
  uint32_t acc = M.G.flags[c] ^ M.G.pair_idx[c] ^ M.G.cellid[c];
  for (int w = 0; w < 2; ++w) {
    const uint32_t l = 2 * c + w, n = M.G.L.nrun[l];
    const uint2 *r = M.G.L.pool + M.G.L.off[l];
    acc ^= M.G.L.cap[l] ^ M.G.L.total[l];
    for (uint32_t q = 0; q < n && q < 64; ++q) {
      const uint32_t v = r[q].x;
      if (v >= M.G.ncp) continue;
      acc ^= M.G.flags[v] ^ M.G.pair_idx[v] ^ M.G.cellid[v];
      for (int u = 0; u < 2; ++u) {
        const uint32_t lv = 2 * v + u;
        acc ^= M.G.L.nrun[lv] ^ M.G.L.cap[lv] ^ M.G.L.total[lv];
        if (M.G.L.nrun[lv]) acc ^= M.G.L.pool[M.G.L.off[lv]].x;
      }
    }
  }
  return acc;
}

__global__ void k_seq_prefetch(const MGraph *graphs, const SeqJob *jobs, uint32_t *sink) {
  const SeqJob jb = jobs[blockIdx.y];
  const MGraph &M = graphs[jb.g0];
  uint32_t acc = 0;
  const long long w = jb.ixn.r - jb.ixn.l + 1, h = jb.ixn.t - jb.ixn.b + 1;
  GRID_LOOP(t, w * h) {
    const uint32_t si = M.find(pack_cellid(jb.ixn.l + (int)(t % w), jb.ixn.b + (int)(t / w)));
    if (si == NO_CP || si >= M.G.ncp) continue;
    acc ^= touch_cp(M, si) ^ touch_cp(M, M.G.pair_idx[si]);
  }
  if (acc == 0x9E3779B9u && sink) *sink = acc;
}

// merge_up's boundary cancellations.  A cancellation reads and writes the lists
// of its two points and of their neighbours, and adds edges among those alone;
// so cells whose pairs' points and neighbours are joined, over the whole
// boundary, by no chain of common points never meet, and each such group can be
// taken on its own, in the loop's order within it.  On white noise most groups
// are a few cells long (2048^2 cut in two: 2,400 cancellations, the longest group
// 220); where one extremum is everybody's neighbour there is one group.
// (2048^2 white noise in 16 pieces, all levels: 12.4 ms as one group per merge,
// 3.0 ms so, finding the groups included; a smooth 1025x769 field, one group: the
// search costs 0.1 ms a level of 4.)
//
// A block takes a group at a time.  Its first warp walks the group's cells in the
// loop's order, 32 at a time: their lanes look the
// cells up side by side (cell -> point -> flags and pair -> the pair's cell)
// and drop those the loop would skip whatever happens before their turn; then
// the cells left are done one after the other (warp_graph.cuh).  A
// cancellation's list edits are shared by SEQ_WARPS warps: the short lists are
// the first warp's, the longer ones go round.  A cancellation is a chain of
// memory round trips (one thread took 19,000 cycles for one on 2048^2 white
// noise; here 5,000), so one more warp runs a batch of cells ahead and brings what
// they will read into L1: their points, both points' lists, the neighbours' list
// descriptors and lists.
constexpr int SEQ_WARPS = 4;
constexpr uint32_t SEQ_STAGE = 512;  // runs of scratch per warp in shared memory
struct SeqShared {
  TeamState team;
  WarpGraph::Pair pair;
  int stop;
  long long at;    // the first warp's batch, as a place in the group
  uint32_t first;  // the group's first place, NO_CP: none left
  uint2 stage[SEQ_WARPS * SEQ_STAGE];
};
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// Into L1: point c's lists, and the flags, list descriptors and first list
// line of their first neighbours.
__device__ __forceinline__ void warm_point(const MGraph &M, uint32_t c) {
  const uint2 off = reinterpret_cast<const uint2 *>(M.G.L.off)[c], n = reinterpret_cast<const uint2 *>(M.G.L.nrun)[c];
  prefetch_l1(M.G.L.total + 2 * c);
  constexpr uint32_t Q = 12;
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const uint2 *r = M.G.L.pool + (w ? off.y : off.x);
    const uint32_t m = w ? n.y : n.x;
    uint32_t v[Q], o[Q];
#pragma unroll
    for (uint32_t q = 0; q < Q; ++q) v[q] = q < m ? r[q].x : M.G.ncp;
#pragma unroll
    for (uint32_t q = 0; q < Q; ++q) {
      o[q] = 0;
      if (v[q] < M.G.ncp) {
        o[q] = M.G.L.off[2 * v[q] + 1 - w];
        prefetch_l1(M.G.flags + v[q]);
        prefetch_l1(M.G.L.nrun + 2 * v[q]);
        prefetch_l1(M.G.L.cap + 2 * v[q]);
        prefetch_l1(M.G.L.total + 2 * v[q]);
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < Q; ++q)
      if (v[q] < M.G.ncp) prefetch_l1(M.G.L.pool + o[q]);
  }
}

// Whether the loop would act on the point si of cell (x, y) with partner pi.
__device__ __forceinline__ bool cell_acts(const MGraph &M, int x, int y, uint32_t pi) {
  const uint32_t p = M.G.cellid[pi];
  return (M.rect.interior(x, y) || M.ext.boundary(x, y)) && (M.rect.interior(px_(p), py_(p)) || M.ext.boundary(px_(p), py_(p)));
}

// Cell t of the boundary, for merge_up: its point si and partner pi; 1 where
// the loop may act at its turn, 0 where it passes, 2 no point there, 3 a
// partner outside the complex.  (A cell already cancelled, or not
// boundary-cancelable, stays so.)
__device__ __forceinline__ int up_cell(const MGraph &M, const CRect &ixn, long long w, long long t, uint32_t &si, uint32_t &pi) {
  const int x = ixn.l + (int)(t % w), y = ixn.b + (int)(t / w);
  si = M.find(pack_cellid(x, y));
  if (si >= M.G.ncp) return 2;
  const uint8_t f = M.G.flags[si];
  pi = M.G.pair_idx[si];
  if (!(f & F_BCANCEL) || (f & F_CANCELLED)) return 0;
  return pi >= M.G.ncp ? 3 : cell_acts(M, x, y, pi) ? 1 : 0;
}
__device__ __forceinline__ void seq_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * SEQ_WARPS) : "memory"); }

// The groups of a job's boundary cells: cells [base, base + n) of the arrays
// that all jobs share.
struct UpWork {
  uint32_t *slot;           // per critical point: the first cell that has it in its reach (null: no groups)
  unsigned long long *top;  // the list pool's top
  uint32_t *ctr;            // [0] groups, [1] groups taken, [2] 1: no groups, all cells in order, [3] blocks done
  uint32_t base, n;
};
struct UpGroups {
  const UpWork *work;
  uint32_t *parent;       // union-find over a job's cells; NO_CP: the cell never acts
  uint32_t *key, *cell;   // a place's group (its first cell, over all jobs) and cell, sorted by group; key = total: never acts
  uint32_t *first;        // per job from base on: the groups' first places, in no order
  uint32_t total;
};
constexpr int UP_BLOCKS = 64;  // blocks per job

// The root of cell a; every step leaves a shortcut.  Parents only get smaller.
__device__ __forceinline__ uint32_t group_of(uint32_t *parent, uint32_t a) {
  volatile uint32_t *const p = parent;
  for (;;) {  // (a falls with every step)
    const uint32_t b = p[a];
    if (b >= a) return a;
    const uint32_t c = p[b];
    if (c < b) p[a] = c;
    a = b;
  }
}
__device__ __forceinline__ bool join_groups(uint32_t *parent, uint32_t a, uint32_t b) {
  for (int guard = 0; guard < 1 << 20; ++guard) {  // (a failed CAS: the other thread's succeeded)
    a = group_of(parent, a);
    b = group_of(parent, b);
    if (a == b) return true;
    if (a > b) { const uint32_t c = a; a = b; b = c; }
    if (atomicCAS(&parent[b], b, a) == b) return true;
  }
  return false;
}
__global__ void k_up_init(const MGraph *graphs, const SeqJob *jobs, UpGroups g) {
  const UpWork w = g.work[blockIdx.y];
  GRID_LOOP(t, (long long)w.n) g.parent[w.base + t] = (uint32_t)t;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *w.top = graphs[jobs[blockIdx.y].g0].G.L.top;
    if (!w.slot) w.ctr[2] = 1;
  }
}
// A warp per cell: a cell that may act leaves its number at its reach and is
// joined with the cells that were there, one of each of their groups (32 cells a
// warp and a join per point took 320 us on a smooth field's 2049 cells).
__global__ void k_up_join(const MGraph *graphs, const SeqJob *jobs, UpGroups g) {
  const UpWork wk = g.work[blockIdx.y];
  const SeqJob jb = jobs[blockIdx.y];
  const MGraph &M = graphs[jb.g0];
  const int lane = threadIdx.x & 31;
  const long long w = jb.ixn.r - jb.ixn.l + 1;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  uint32_t *const parent = g.parent + wk.base;
  bool lost = false;
  for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < wk.n; t += warps) {
    uint32_t c[2] = {0, 0};
    const int what = up_cell(M, jb.ixn, w, t, c[0], c[1]);
    if (what > 1) lost = true;  // an error at its turn: the plain order
    if (what == 0) parent[t] = NO_CP;
    if (what != 1) continue;
    auto reach = [&](bool on, uint32_t v) {
      uint32_t old = t;
      if (on && v < M.G.ncp) {
        const uint32_t o = atomicMin(&wk.slot[v], t);
        if (o != NO_CP) old = o;
      }
      for (int guard = 0;; ++guard) {
        const uint32_t r = group_of(parent, old), own = group_of(parent, t);
        const unsigned apart = __ballot_sync(FULL_WARP, r != own);
        if (!apart) break;
        if (guard == 4096) { lost = true; break; }  // (others' joins may show roots apart that are not)
        if (lane == __ffs(apart) - 1 && !join_groups(parent, r, own)) lost = true;
        __syncwarp();
      }
    };
    reach(lane < 2, c[lane & 1]);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t q = 2 * c[l >> 1] + (l & 1), m = M.G.L.nrun[q];
      const uint2 *r = M.G.L.pool + M.G.L.off[q];
      for (uint32_t k0 = 0; k0 < m; k0 += 32) reach(k0 + lane < m, k0 + lane < m ? r[k0 + lane].x : 0);
    }
  }
  if (lost) wk.ctr[2] = 1;
}
__global__ void k_up_key(UpGroups g) {
  const UpWork w = g.work[blockIdx.y];
  GRID_LOOP(t, (long long)w.n) {
    g.key[w.base + t] = g.parent[w.base + t] == NO_CP ? g.total : w.base + group_of(g.parent + w.base, (uint32_t)t);
    g.cell[w.base + t] = (uint32_t)t;
  }
}
__global__ void k_up_first(UpGroups g, int njobs) {
  GRID_LOOP(q, (long long)g.total) {
    const uint32_t k = g.key[q];
    if (k >= g.total || (q > 0 && g.key[q - 1] == k)) continue;
    int b = 0;  // the last job that starts at or before cell k
    for (int hi = njobs - 1; b < hi;) {
      const int m = (b + hi + 1) >> 1;
      if (g.work[m].base <= k) b = m; else hi = m - 1;
    }
    g.first[g.work[b].base + atomicAdd(g.work[b].ctr, 1u)] = (uint32_t)q;
  }
}

__global__ void __launch_bounds__(32 * (SEQ_WARPS + 1), 1) k_merge_up_seq(MGraph *graphs, const SeqJob *jobs, UpGroups g, uint32_t *status) {
  __shared__ SeqShared sh;
  const SeqJob jb = jobs[blockIdx.y];
  const UpWork wk = g.work[blockIdx.y];
  const bool plain = wk.ctr[2] != 0;  // all cells in order, by the job's first block
  const MGraph M = graphs[jb.g0];     // (a copy of the descriptor: pointers stay in registers)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long w = jb.ixn.r - jb.ixn.l + 1;
  WarpGraph W;
  W.G = M.G;
  W.lane = lane;
  W.team = &sh.team;
  W.stage = sh.stage + (warp % SEQ_WARPS) * SEQ_STAGE;
  W.nstage = SEQ_STAGE;
  W.G.tmp_cap = M.G.tmp_cap / (SEQ_WARPS * gridDim.x);
  W.G.tmp = M.G.tmp + (blockIdx.x * SEQ_WARPS + warp % SEQ_WARPS) * W.G.tmp_cap;
  if (threadIdx.x == 0) {
    sh.team.shared_top = wk.top;
    sh.team.fail = 0;
    sh.stop = 0;
  }
  for (bool more = !plain || blockIdx.x == 0; more;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      sh.at = 0;
      sh.first = 0;
      if (!plain && !sh.team.fail) {
        const uint32_t q = atomicAdd(wk.ctr + 1, 1u);
        sh.first = q < wk.ctr[0] ? g.first[wk.base + q] : NO_CP;
      }
      if (sh.team.fail || sh.stop == 2) sh.first = NO_CP;
      sh.stop = 0;
    }
    __syncthreads();
    const uint32_t first = sh.first, key = plain || first == NO_CP ? 0 : g.key[first];
    if (first == NO_CP) break;
    more = !plain;
    // the group's cell at place k, -1 past its end
    auto cell_at = [&](long long k) -> long long {
      if (plain) return k < wk.n ? k : -1;
      return first + k < g.total && g.key[first + k] == key ? (long long)g.cell[first + k] : -1;
    };
    if (warp == SEQ_WARPS) {  // reads ahead: at most one batch beyond the first warp's
      for (long long t0 = 0;; t0 += 32) {
        const long long t = cell_at(t0 + lane);
        if (!__any_sync(FULL_WARP, t >= 0)) break;
        for (long long polls = 0; *(volatile long long *)&sh.at + 32 < t0 && !*(volatile int *)&sh.stop && polls < (1ll << 26); ++polls) __nanosleep(200);
        if (__any_sync(FULL_WARP, *(volatile int *)&sh.stop)) break;
        uint32_t si = 0, pi = 0;
        if (t >= 0 && up_cell(M, jb.ixn, w, t, si, pi) == 1) {
          warm_point(M, si);
          warm_point(M, pi);
        }
        __syncwarp();
      }
      continue;
    }
    if (warp > 0) {
      for (;;) {
        seq_barrier();
        if (sh.stop) break;
        if (warp == SEQ_WARPS - 1) W.close(sh.pair, 0);  // (nobody reads what it changes until the next pair)
        W.edit_neighbours(sh.pair, warp, SEQ_WARPS);
        if (W.G.fail) sh.team.fail = 1;
        seq_barrier();
      }
      continue;
    }
    int stop = 0;
    for (long long t0 = 0; !stop; t0 += 32) {
      if (lane == 0) *(volatile long long *)&sh.at = t0;
      uint32_t si = 0, pi = 0;
      const long long t = cell_at(t0 + lane);
      if (!__any_sync(FULL_WARP, t >= 0)) break;
      const int todo = t >= 0 ? up_cell(M, jb.ixn, w, t, si, pi) : 0;
      __syncwarp();
      for (unsigned left = __ballot_sync(FULL_WARP, todo != 0); left && !stop; left &= left - 1) {
        const int s = __ffs(left) - 1;
        const int what = __shfl_sync(FULL_WARP, todo, s);
        const uint32_t c = __shfl_sync(FULL_WARP, si, s), d = __shfl_sync(FULL_WARP, pi, s);
        if (what != 2 && (M.G.flags[c] & F_CANCELLED)) continue;  // with an earlier cell
        if (what != 1) {  // "missing common bndry cp", or a partner outside the complex
          if (lane == 0) set_status(status, ST_INVARIANT);
          stop = 2;
          break;
        }
        WarpGraph::Pair q{reinterpret_cast<const uint2 *>(M.G.L.off)[c], reinterpret_cast<const uint2 *>(M.G.L.off)[d],
                          reinterpret_cast<const uint2 *>(M.G.L.nrun)[c], reinterpret_cast<const uint2 *>(M.G.L.nrun)[d], c, d};
        if (!W.orient(q)) continue;
        if (lane == 0) sh.pair = q;
        seq_barrier();
        W.edit_neighbours(q, 0, SEQ_WARPS);
        if (W.G.fail) sh.team.fail = 1;
        seq_barrier();
        if (sh.team.fail) stop = 2;
      }
    }
    if (lane == 0) *(volatile int *)&sh.stop = stop ? stop : 1;
    __syncwarp();
    seq_barrier();
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (sh.team.fail) set_status(status, ST_SIMPLIFY_LIMIT);
  if (atomicAdd(wk.ctr + 3, 1u) + 1 == gridDim.x) graphs[jb.g0].G.L.top = atomicAdd(wk.top, 0ull);
}

// merge_down's boundary uncancellations, one job per block.  The loop runs in
// reverse row-major order over the cells whose point is cancelled; a pair's
// two lists are rewritten from lists of pairs uncancelled before it, so the
// block's warps take them in the loop's order and wait only for the lists
// their own name (WarpGraph::uncancel_shared).  Before that the whole block
// lists the pairs: a pair with both points on the boundary belongs to the cell
// the loop meets first.  A pair whose points do not name each other takes the
// job to the plain order on one warp.  (2048^2 white noise in 16 pieces, all
// levels: 19.5 ms on one thread, 1.6 ms here.)
constexpr int DOWN_WARPS = 16;
constexpr uint32_t DOWN_STAGE = 512, DOWN_SHARED = 4096;  // runs of scratch: each warp's own, the one they share
struct DownWork {
  uint32_t *ord;  // per point of the job's graph (zeroed)
  uint2 *pairs;   // room for the boundary's cells
};
constexpr int DOWN_CELLS = 32768;  // cell coordinates are below 2^15, and a boundary is one cell wide
constexpr uint32_t DOWN_DONE = 2 * DOWN_CELLS / 32;  // words
constexpr size_t DOWN_SMEM = sizeof(uint2) * (DOWN_WARPS * DOWN_STAGE + DOWN_SHARED) + sizeof(uint32_t) * DOWN_DONE;
__global__ void __launch_bounds__(32 * DOWN_WARPS, 1) k_merge_down_seq(MGraph *graphs, const SeqJob *jobs, int njobs,
                                                                       const DownWork *works, uint32_t *status) {
  extern __shared__ __align__(16) unsigned char down_smem[];
  __shared__ TeamState team;
  __shared__ uint32_t count[DOWN_WARPS];
  __shared__ int odd;
  const int b = blockIdx.x;
  if (b >= njobs) return;
  const SeqJob jb = jobs[b];
  const MGraph M = graphs[jb.g0];
  const DownWork wk = works[b];
  const int warp = threadIdx.x >> 5;
  WarpGraph W;
  W.G = M.G;
  W.lane = threadIdx.x & 31;
  W.team = &team;
  uint2 *buf = reinterpret_cast<uint2 *>(down_smem);
  W.stage = buf + (size_t)warp * DOWN_STAGE;
  W.nstage = DOWN_STAGE;
  W.shared_stage = buf + DOWN_WARPS * DOWN_STAGE;
  W.nshared_stage = DOWN_SHARED;
  W.done = reinterpret_cast<uint32_t *>(W.shared_stage + DOWN_SHARED);
  for (uint32_t i = threadIdx.x; i < DOWN_DONE; i += blockDim.x) W.done[i] = 0;
  const long long w = jb.ixn.r - jb.ixn.l + 1, n = w * (jb.ixn.t - jb.ixn.b + 1);
  if (threadIdx.x == 0) {
    team.top = M.G.L.top;
    team.shared_top = nullptr;
    team.fail = team.wrong = team.late = team.beat = 0;
    team.lock = 0;
    odd = n > DOWN_CELLS;
  }
  __syncthreads();
  // cell t's point si and its partner pi: 1 where the loop acts on them, 0
  // where it passes, 2 no point there, 3 a partner outside the complex
  auto cell = [&](long long t, uint32_t &si, uint32_t &pi) -> int {
    const int x = jb.ixn.l + (int)(t % w), y = jb.ixn.b + (int)(t / w);
    si = M.find(pack_cellid(x, y));
    if (si >= M.G.ncp) return 2;
    if (!(M.G.flags[si] & F_CANCELLED)) return 0;
    pi = M.G.pair_idx[si];
    return pi >= M.G.ncp ? 3 : cell_acts(M, x, y, pi) ? 1 : 0;
  };
  uint32_t si = 0, pi = 0;
  for (long long t = threadIdx.x; t < n; t += blockDim.x) {
    const int what = cell(t, si, pi);
    if (what == 1) {
      atomicMax(&wk.ord[si], (uint32_t)t + 1);
      atomicMax(&wk.ord[pi], (uint32_t)t + 1);
      if (M.G.pair_idx[pi] != si) odd = 1;
    }
    if (what == 2) team.wrong = 1;  // "missing common bndry cp"
    if (what == 3) odd = 1;
  }
  __syncthreads();
  if (!team.wrong && !odd) {
    // the pairs in cell order: each warp its part of the boundary
    const long long part = ((n + DOWN_WARPS - 1) / DOWN_WARPS + 31) / 32 * 32, c0 = part * warp, c1 = min(c0 + part, n);
    uint32_t mine = 0;
    for (long long t0 = c0; t0 < c1; t0 += 32) {
      const long long t = t0 + W.lane;
      const bool own = t < c1 && cell(t, si, pi) == 1 && wk.ord[si] == (uint32_t)t + 1;
      mine += __popc(__ballot_sync(FULL_WARP, own));
    }
    if (W.lane == 0) count[warp] = mine;
    __syncthreads();
    uint32_t at = 0, np = 0;
    for (int k = 0; k < DOWN_WARPS; ++k) {
      if (k < warp) at += count[k];
      np += count[k];
    }
    for (long long t0 = c0; t0 < c1; t0 += 32) {
      const long long t = t0 + W.lane;
      const bool own = t < c1 && cell(t, si, pi) == 1 && wk.ord[si] == (uint32_t)t + 1;
      const unsigned m = __ballot_sync(FULL_WARP, own);
      if (own) {
        const uint2 *p = M.G.runs(2 * si);
        uint32_t lo = 0, hi = M.G.L.nrun[2 * si];
        while (lo < hi) {
          const uint32_t c = (lo + hi) >> 1;
          if (p[c].x < pi) lo = c + 1; else hi = c;
        }
        const bool first = lo < M.G.L.nrun[2 * si] && p[lo].x == pi;  // asc(si) holds pi
        wk.pairs[at + __popc(m & W.lt())] = first ? make_uint2(si, pi) : make_uint2(pi, si);
      }
      at += __popc(m);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < np; k += blockDim.x) {
      const uint2 c = wk.pairs[k];
      wk.ord[c.x] = wk.ord[c.y] = k + 1;
    }
    if (threadIdx.x == 0) team.ticket = 2ull * np;
    __syncthreads();
    W.ord = wk.ord;
    W.uncancel_shared(wk.pairs, np);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < np; k += blockDim.x) {
      const uint2 c = wk.pairs[k];
      M.G.flags[c.x] &= ~F_CANCELLED;
      M.G.flags[c.y] &= ~F_CANCELLED;
    }
  } else if (!team.wrong && warp == 0) {
    for (long long t = n - 1; t >= 0 && !team.wrong && !W.G.fail; --t) {
      const int what = cell(t, si, pi);
      if (what >= 2 || (what == 1 && !W.uncancel_pairs(si, pi))) team.wrong = 1;
      if (W.G.fail) team.fail = 1;
      __syncwarp();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    MGraph g = M;
    g.G.fail = team.fail != 0 && !team.wrong;
    g.G.L.top = team.top;
    if (team.late) set_status(status, ST_WAIT_LIMIT);
    else if (team.wrong) set_status(status, ST_INVARIANT);  // (the other warps stopped for it)
    else if (team.fail) set_status(status, ST_SIMPLIFY_LIMIT);
    graphs[jb.g0] = g;
  }
}

// ---------------------------------------------------------------------------
// merge_up's boundary cancellations in ordered-parallel rounds.  Task t is
// cell t of the shared boundary in row-major order.  Each round looks at a
// window: the first `win` cells from the first pending task on.  Every
// pending task of the window reserves its footprint -- the critical points
// whose lists or flags its cancellation reads or writes -- with the
// round-tagged key (round, t) in a per-point slot (atomicMin: the round's
// smallest task touching the point wins); tasks sharing a slot are joined in
// a union-find that hooks the larger root under the smaller; and the root of
// each group, its smallest task, runs.  Every pending task earlier than a
// window task is inside the window, so a root has no earlier pending task
// that overlaps it.  Edges are only added inside a running task's footprint,
// so groups cannot merge through growth and every task sees the graph the
// row-major loop would show it.  The first pending task is always a root, so
// every round commits at least one task.  One block per merge; the rounds are
// separated by barriers of the block.  Each thread allocates list room from
// its own slice of the pool's free part, so the graph code stays that of one
// thread.  Where groups stay large (one point in most footprints, as a large
// extremum on a smooth field), rounds commit few tasks each: after
// ROUND_PATIENCE rounds in a row below `min_commits`, or if a union-find
// guard runs out, thread 0 runs the remaining tasks in row-major order, which
// is exact at any round boundary (every task that ran commutes with every
// earlier one still pending), from a quarter of the free pool kept for it.
// ---------------------------------------------------------------------------
constexpr int ROUND_THREADS = 512, ROUND_TASKS = 32768, ROUND_PATIENCE = 8;
struct RoundSmem {
  uint32_t parent[ROUND_TASKS];
  uint32_t done[ROUND_TASKS / 32];
};

// Parents only point to smaller tasks of the window, so a chain is shorter
// than the window and the guard never ends a search early.
__device__ __forceinline__ uint32_t uf_root(uint32_t *parent, uint32_t a) {
  for (int guard = 0; guard < ROUND_TASKS; ++guard) {
    const uint32_t p = ((volatile uint32_t *)parent)[a];
    if (p == a) return a;
    a = p;
  }
  return a;
}
// False if the join did not happen within the guard (each failed CAS means
// another thread hooked a root meanwhile); the caller then stops the rounds.
__device__ __forceinline__ bool uf_join(uint32_t *parent, uint32_t a, uint32_t b) {
  for (int guard = 0; guard < 4 * ROUND_TASKS; ++guard) {
    a = uf_root(parent, a);
    b = uf_root(parent, b);
    if (a == b) return true;
    if (a > b) { const uint32_t t = a; a = b; b = t; }
    if (atomicCAS(&parent[b], b, a) == b) return true;
  }
  return false;
}

// The cell's point and, while it may still cancel, its partner and both
// points' neighbours.
template <class F>
__device__ void up_footprint(const MGraph &M, uint32_t si, F f) {
  f(si);
  const uint8_t fl = M.G.flags[si];
  if ((fl & F_CANCELLED) || !(fl & F_BCANCEL)) return;
  const uint32_t pi = M.G.pair_idx[si];
  if (pi >= M.G.ncp) return;
  f(pi);
  const uint32_t c2[2] = {si, pi};
  for (int k = 0; k < 2; ++k)
    for (int w = 0; w < 2; ++w) {
      const uint32_t l = 2 * c2[k] + w, n = M.G.L.nrun[l];
      const uint2 *r = M.G.L.pool + M.G.L.off[l];
      for (uint32_t q = 0; q < n; ++q) f(r[q].x);
    }
}

// Whether cell (x, y) can ever act: the rect / ext test of the loop on it and
// its partner (fixed for the whole loop; flags are not).
__device__ __forceinline__ bool up_cell_static(const MGraph &M, int x, int y, uint32_t si) {
  if (si >= M.G.ncp) return true;  // left to the loop body, which reports it
  const uint32_t pi = M.G.pair_idx[si];
  if (pi >= M.G.ncp) return true;
  const uint32_t p = M.G.cellid[pi];
  return (M.rect.interior(x, y) || M.ext.boundary(x, y)) && (M.rect.interior(px_(p), py_(p)) || M.ext.boundary(px_(p), py_(p)));
}

// The first task at or after `from` whose done bit is clear (n if none),
// into *lo (which the caller set to n); all threads take part.
__device__ __forceinline__ void first_pending(const RoundSmem &S, long long from, long long n, unsigned int *lo) {
  const long long nw = (n + 31) / 32;
  for (long long wi = from / 32 + threadIdx.x; wi < nw; wi += blockDim.x) {
    uint32_t open = ~S.done[wi];
    if (wi == from / 32) open &= ~0u << (from & 31);
    if (wi == nw - 1 && (n & 31)) open &= (1u << (n & 31)) - 1;
    if (open) atomicMin(lo, (unsigned int)(wi * 32 + __ffs(open) - 1));
  }
}

__global__ void __launch_bounds__(ROUND_THREADS, 1) k_merge_up_rounds(MGraph *graphs, const SeqJob *jobs, int njobs,
                                                                      unsigned long long *const *slots, uint32_t *status) {
  extern __shared__ __align__(16) unsigned char round_smem[];
  RoundSmem &S = *reinterpret_cast<RoundSmem *>(round_smem);
  __shared__ int abort_all, uf_bad;
  __shared__ unsigned int lo_s, commits;
  const int b = blockIdx.x;
  if (b >= njobs) return;
  const SeqJob jb = jobs[b];
  MGraph g = graphs[jb.g0];  // every thread's own descriptor copy, read before any write-back
  const long long w = jb.ixn.r - jb.ixn.l + 1, h = jb.ixn.t - jb.ixn.b + 1, n = w * h;
  unsigned long long *slot = slots[b];
  if (n > ROUND_TASKS || !slot || jb.win <= 0) {  // one thread
    if (threadIdx.x == 0) {
      merge_up_cancel(g, jb.ixn, status);
      if (g.G.fail) set_status(status, ST_SIMPLIFY_LIMIT);
      graphs[jb.g0] = g;
    }
    return;
  }
  const long long win = jb.win < ROUND_TASKS ? jb.win : ROUND_TASKS;
  if (threadIdx.x == 0) { abort_all = 0; uf_bad = 0; lo_s = (unsigned int)n; }
  for (long long t = threadIdx.x; t < ROUND_TASKS / 32; t += blockDim.x) S.done[t] = 0;
  __syncthreads();
  const unsigned long long free_runs = g.G.L.pool_cap - g.G.L.top, pool_end = g.G.L.pool_cap;
  const unsigned long long room = (free_runs - free_runs / 4) / blockDim.x, fin_start = g.G.L.top + room * blockDim.x;
  const unsigned long long tmp_cap0 = g.G.tmp_cap;
  g.G.L.top += room * threadIdx.x;  // this thread's slice of the free pool
  g.G.L.pool_cap = g.G.L.top + room;
  g.G.tmp_cap = 0;  // no shared scratch: cancel_pairs takes its per-entry path (the same result)
  auto cell_of = [&](long long t, int &x, int &y) { x = jb.ixn.l + (int)(t % w); y = jb.ixn.b + (int)(t / w); };
  auto is_done = [&](long long t) { return (S.done[t >> 5] >> (t & 31)) & 1u; };
  // cells that can never act are done from the start
  for (long long t = threadIdx.x; t < n; t += blockDim.x) {
    int x, y;
    cell_of(t, x, y);
    const uint32_t si = g.find(pack_cellid(x, y));
    if (si != NO_CP && !up_cell_static(g, x, y, si)) atomicOr(&S.done[t >> 5], 1u << (t & 31));
  }
  __syncthreads();
  first_pending(S, 0, n, &lo_s);
  __syncthreads();
  int slow = 0;  // rounds in a row that committed fewer than min_commits tasks
  for (uint32_t round = 0; round < (uint32_t)n + 1; ++round) {
    const long long lo = lo_s;
    if (lo >= n || abort_all || uf_bad || slow >= ROUND_PATIENCE) break;
    const long long hi = lo + win < n ? lo + win : n;
    const unsigned long long tag = (unsigned long long)(0xFFFFFFFFu - round) << 32;
    __syncthreads();  // every thread has read lo_s and the flags
    if (threadIdx.x == 0) { commits = 0; lo_s = (unsigned int)n; }
    // reserve
    for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
      if (is_done(t)) continue;
      S.parent[t] = (uint32_t)t;
      int x, y;
      cell_of(t, x, y);
      const uint32_t si = g.find(pack_cellid(x, y));
      if (si >= g.G.ncp) continue;  // the loop body reports it when the task runs
      up_footprint(g, si, [&](uint32_t c) { if (c < g.G.ncp) atomicMin(&slot[c], tag | (unsigned long long)t); });
    }
    __syncthreads();
    // join the tasks that share a point
    for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
      if (is_done(t)) continue;
      int x, y;
      cell_of(t, x, y);
      const uint32_t si = g.find(pack_cellid(x, y));
      if (si >= g.G.ncp) continue;
      up_footprint(g, si, [&](uint32_t c) {
        if (c >= g.G.ncp) return;
        const unsigned long long v = slot[c];
        if ((v & 0xFFFFFFFF00000000ull) == tag && (v & 0xFFFFFFFFull) < (unsigned long long)n)
          if (!uf_join(S.parent, (uint32_t)t, (uint32_t)(v & 0xFFFFFFFFull))) uf_bad = 1;
      });
    }
    __syncthreads();
    // the smallest task of each group runs (none if a join was lost)
    if (!uf_bad)
      for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
        if (is_done(t) || uf_root(S.parent, (uint32_t)t) != (uint32_t)t) continue;
        int x, y;
        cell_of(t, x, y);
        if (!merge_up_cell(g, x, y, status) || g.G.fail) abort_all = 1;
        atomicOr(&S.done[t >> 5], 1u << (t & 31));
        atomicAdd(&commits, 1u);
      }
    __syncthreads();
    first_pending(S, lo, n, &lo_s);
    __syncthreads();
    slow = commits < (unsigned int)jb.min_commits ? slow + 1 : 0;
  }
  if (g.G.fail) set_status(status, ST_SIMPLIFY_LIMIT);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!abort_all) {  // tasks left to one thread, in row-major order
      MGraph f = g;
      f.G.L.top = fin_start;
      f.G.L.pool_cap = pool_end;
      f.G.tmp_cap = tmp_cap0;
      f.G.fail = false;
      for (long long t = 0; t < n && !f.G.fail; ++t) {
        if (is_done(t)) continue;
        int x, y;
        cell_of(t, x, y);
        if (!merge_up_cell(f, x, y, status)) break;
      }
      if (f.G.fail) set_status(status, ST_SIMPLIFY_LIMIT);
    }
    // the slices are used up: later allocations of this graph find no room
    g.G.L.top = pool_end;
    g.G.L.pool_cap = pool_end;
    g.G.tmp_cap = tmp_cap0;
    graphs[jb.g0] = g;
  }
}

MGraph &mg(MGraphHost &h) { return *reinterpret_cast<MGraph *>(h.raw); }

// List pool (runs) beyond the lists themselves for the steps
// along a shared boundary: lists there relocate to the pool top as they
// grow (the graphs start without slack); retries multiply it.
unsigned long long boundary_room(const int ixn[4]) {
  const unsigned long long cells = (unsigned long long)(ixn[2] - ixn[0] + 1) * (ixn[3] - ixn[1] + 1);
  return (1ull << 20) + 256ull * cells;
}

double now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Runs the jobs side by side and brings the graphs' counters back; adds its
// wall time to *ms.  merge_up's blocks of one job take groups of cells from a
// counter, share the list pool's top (an atomic, UpWork::top) and have a slice
// of the graph's scratch per warp.
cudaError_t run_seq(std::vector<MGraphHost *> &graphs, const std::vector<SeqJob> &jobs, uint32_t *status,
                    cudaStream_t st, double *ms) {
  if (jobs.empty()) return cudaSuccess;
  cudaStreamSynchronize(st);
  const double t0 = now_ms();
  struct Acc {
    double *ms, t0;
    ~Acc() { if (ms) *ms += now_ms() - t0; }
  } acc{ms, t0};
  const size_t ng = graphs.size();
  char *buf = nullptr;
  const size_t nj = jobs.size();
  const size_t gb = sizeof(MGraph) * ng, jbytes = sizeof(SeqJob) * nj;
  // merge_up's jobs in rounds (a window set): per job a slot per critical point
  // of its graph (round-tagged keys, all ones = empty).  merge_down: per job an
  // order word per critical point (zero), then the boundary's pairs.
  const bool down = jobs[0].kind == SEQ_DOWN_BOUNDARY, rounds = !down && jobs[0].win > 0;
  std::vector<size_t> soff(nj, 0), poff(nj, 0);
  size_t sbytes = 0;
  for (size_t k = 0; k < nj && (rounds || down); ++k) {
    soff[k] = sbytes;
    sbytes += (rounds ? 8ull : 4ull) * ((mg(*graphs[jobs[k].g0]).G.ncp + 1 + 31) / 32 * 32);
  }
  const size_t obytes = sbytes;
  for (size_t k = 0; k < nj && down; ++k) {
    const CRect &x = jobs[k].ixn;
    poff[k] = sbytes;
    sbytes += sizeof(uint2) * ((size_t)(x.r - x.l + 1) * (x.t - x.b + 1) + 15) / 16 * 16;
  }
  // merge_up's jobs in groups: per job a slot per critical point; over all jobs
  // six words per boundary cell; a pool top and four counters per job
  const bool groups = !down && !rounds;
  size_t slot_bytes = 0, cells = 0;
  std::vector<size_t> base(nj, 0);
  for (size_t k = 0; k < nj && groups; ++k) {
    const CRect &x = jobs[k].ixn;
    soff[k] = slot_bytes;
    base[k] = cells;
    slot_bytes += 4ull * ((mg(*graphs[jobs[k].g0]).G.ncp + 1 + 31) / 32 * 32);
    cells += (size_t)(x.r - x.l + 1) * (x.t - x.b + 1);
  }
  const size_t cell_bytes = (24 * cells + 15) / 16 * 16;
  if (groups) sbytes = cell_bytes + 32 * nj + slot_bytes;
  const size_t head = (gb + 15) / 16 * 16 + (jbytes + 15) / 16 * 16;
  const size_t pbytes = ((rounds ? 8ull : down ? sizeof(DownWork) : sizeof(UpWork)) * nj + 15) / 16 * 16;
  cudaError_t e = cudaMallocAsync((void **)&buf, head + pbytes + sbytes + 64, st);
  if (e == cudaErrorMemoryAllocation && groups) {  // no room for the slots: all cells in order
    cudaGetLastError();
    sbytes -= slot_bytes;
    slot_bytes = 0;
    e = cudaMallocAsync((void **)&buf, head + pbytes + sbytes + 64, st);
  }
  if (e != cudaSuccess) return e;
  MGraph *dg = (MGraph *)buf;
  SeqJob *dj = (SeqJob *)(buf + ((gb + 15) / 16) * 16);
  unsigned long long **dslot = (unsigned long long **)(buf + head);
  unsigned long long *slots = (unsigned long long *)(buf + head + pbytes);
  std::vector<MGraph> hg(ng);
  for (size_t i = 0; i < ng; ++i) hg[i] = mg(*graphs[i]);
  e = cudaMemcpyAsync(dg, hg.data(), gb, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dj, jobs.data(), jbytes, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && rounds) {
    std::vector<unsigned long long *> hp(nj);
    for (size_t k = 0; k < nj; ++k) hp[k] = slots + soff[k] / 8;
    e = cudaMemcpyAsync(dslot, hp.data(), 8ull * nj, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(slots, 0xFF, sbytes, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // hp is read before it goes out of scope
  }
  if (e == cudaSuccess && down) {
    char *base = buf + head + pbytes;
    std::vector<DownWork> hw(nj);
    for (size_t k = 0; k < nj; ++k) hw[k] = DownWork{(uint32_t *)(base + soff[k]), (uint2 *)(base + poff[k])};
    e = cudaMemcpyAsync(buf + head, hw.data(), sizeof(DownWork) * nj, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(base, 0, obytes, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // hw is read before it goes out of scope
  }
  UpGroups ug{};
  if (e == cudaSuccess && groups) {
    char *const words = buf + head + pbytes, *const ctr = words + cell_bytes, *const slot = ctr + 32 * nj;
    uint32_t *const at = (uint32_t *)words;
    ug = UpGroups{(const UpWork *)(buf + head), at, at + cells, at + 2 * cells, at + 3 * cells, (uint32_t)cells};
    std::vector<UpWork> hw(nj);
    for (size_t k = 0; k < nj; ++k)
      hw[k] = UpWork{slot_bytes ? (uint32_t *)(slot + soff[k]) : nullptr, (unsigned long long *)(ctr + 32 * k),
                     (uint32_t *)(ctr + 32 * k + 8), (uint32_t)base[k],
                     (uint32_t)((k + 1 < nj ? base[k + 1] : cells) - base[k])};
    e = cudaMemcpyAsync(buf + head, hw.data(), sizeof(UpWork) * nj, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(ctr, 0, 32 * nj, st);
    if (e == cudaSuccess && slot_bytes) e = cudaMemsetAsync(slot, 0xFF, slot_bytes, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // hw is read before it goes out of scope
  }
  if (e == cudaSuccess) {
    k_seq_prefetch<<<dim3(64, (unsigned)nj), 256, 0, st>>>(dg, dj, nullptr);
    if (rounds) {
      static SmemLimit limit;
      e = limit.raise(sizeof(RoundSmem), k_merge_up_rounds);
      if (e == cudaSuccess)
        k_merge_up_rounds<<<(unsigned)nj, ROUND_THREADS, sizeof(RoundSmem), st>>>(dg, dj, (int)nj, dslot, status);
    } else if (down) {
      static SmemLimit limit;
      e = limit.raise(DOWN_SMEM, k_merge_down_seq);
      if (e == cudaSuccess)
        k_merge_down_seq<<<(unsigned)nj, 32 * DOWN_WARPS, DOWN_SMEM, st>>>(dg, dj, (int)nj, (const DownWork *)(buf + head), status);
    } else {
      const dim3 grid(32, (unsigned)nj);
      k_up_init<<<grid, 256, 0, st>>>(dg, dj, ug);
      DMSC_LAUNCHED(1);
      if (slot_bytes) {
        k_up_join<<<dim3(256, (unsigned)nj), 256, 0, st>>>(dg, dj, ug);
        k_up_key<<<grid, 256, 0, st>>>(ug);
        int bits = 1;
        while (bits < 32 && (ug.total >> bits)) ++bits;
        e = radix_sort_pairs(ug.key, ug.cell, ug.first + cells, ug.first + 2 * cells, (long long)cells, bits, st);
        k_up_first<<<64, 256, 0, st>>>(ug, (int)nj);
        DMSC_LAUNCHED(3);
      }
      if (e == cudaSuccess)
        k_merge_up_seq<<<dim3(slot_bytes ? UP_BLOCKS : 1, (unsigned)nj), 32 * (SEQ_WARPS + 1), 0, st>>>(dg, dj, ug, status);
    }
    DMSC_LAUNCHED(2);
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(hg.data(), dg, gb, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess)
    for (size_t i = 0; i < ng; ++i) mg(*graphs[i]) = hg[i];
  cudaFreeAsync(buf, st);
  return e;
}

struct Scratch {  // one device allocation carved into arrays
  char *buf = nullptr;
  std::vector<size_t> sz;
  std::vector<void *> ptr;
  cudaError_t alloc(cudaStream_t st) {
    size_t tot = 0;
    for (size_t s : sz) tot += (s + 255) / 256 * 256;
    cudaError_t e = cudaMallocAsync((void **)&buf, tot + 256, st);
    if (e != cudaSuccess) { buf = nullptr; return e; }
    char *p = buf;
    for (size_t s : sz) { ptr.push_back(p); p += (s + 255) / 256 * 256; }
    return cudaSuccess;
  }
  void free(cudaStream_t st) {
    if (buf) cudaFreeAsync(buf, st);
    buf = nullptr;
  }
};

CsrOut csr_out(dmsc_msc &m) {
  return CsrOut{m.cellid.p, m.pair_idx.p, m.aoff.p, m.asc.p, m.doff.p, m.des.p, m.fn.p, m.flags.p};
}

// merge_up of one pair into o's CSR arrays (before the boundary cancellations);
// *tab receives the cell table of the result over O.bbox (the caller owns it).
cudaError_t union_one(const dmsc_msc &A, const dmsc_msc &B, dmsc_msc &O, CRect ixn, uint32_t *status, uint32_t **tab,
                      cudaStream_t st) {
  const long long nA = A.ncp, nB = B.ncp, bound = nA + nB;
  if (bound >= (1ll << 30) || A.nasc + B.nasc >= (1ll << 32) - 1 || A.ndes + B.ndes >= (1ll << 32) - 1)
    return cudaErrorInvalidValue;  // 32-bit indices and offsets
  const int tw = O.bbox[2] - O.bbox[0] + 1, th = O.bbox[3] - O.bbox[1] + 1;
  if (tw <= 0 || th <= 0) return cudaErrorInvalidValue;
  const size_t tcells = (size_t)tw * th;
  cudaError_t e = cudaMallocAsync((void **)tab, sizeof(uint32_t) * tcells, st);
  if (e != cudaSuccess) { *tab = nullptr; return e; }
  e = cudaMemsetAsync(*tab, 0xFF, sizeof(uint32_t) * tcells, st);
  if (e == cudaSuccess) e = O.cellid.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.fn.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.pair_idx.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.flags.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.aoff.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.doff.ensure(bound + 1, st);
  if (e == cudaSuccess) e = O.asc.ensure(A.nasc + B.nasc + 1, st);
  if (e == cudaSuccess) e = O.des.ensure(A.ndes + B.ndes + 1, st);
  if (e != cudaSuccess) return e;
  Scratch s;
  // keepA, idxA, idxB, isnew, posB, tot_a, tot_d, mix, counters
  s.sz = {4ull * (nA + 1), 4ull * (nA + 1), 4ull * (nB + 1), 4ull * (nB + 1), 4ull * (nB + 1),
          4ull * (bound + 1), 4ull * (bound + 1), (size_t)bound + 1, 64};
  if (e == cudaSuccess) e = s.alloc(st);
  if (e != cudaSuccess) return e;
  uint32_t *keep = (uint32_t *)s.ptr[0], *idxA = (uint32_t *)s.ptr[1], *idxB = (uint32_t *)s.ptr[2];
  uint32_t *isnew = (uint32_t *)s.ptr[3], *posB = (uint32_t *)s.ptr[4];
  CellTab H{*tab, O.bbox[0], O.bbox[1], tw, th};
  uint32_t *tot_a = (uint32_t *)s.ptr[5], *tot_d = (uint32_t *)s.ptr[6];
  uint8_t *mix = (uint8_t *)s.ptr[7];
  uint32_t *cnt = (uint32_t *)s.ptr[8];  // [0] kept of A, [1] new of B
  const CsrIn a = csr_in(A), b = csr_in(B);
  CsrOut o = csr_out(O);
  if (e == cudaSuccess) e = cudaMemsetAsync(tot_a, 0, 4ull * (bound + 1), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(tot_d, 0, 4ull * (bound + 1), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(mix, 0, bound + 1, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, 64, st);
  // union (:56-75)
  if (e == cudaSuccess && nA) {
    k_keep<<<nblk(nA), 256, 0, st>>>(a, keep);
    DMSC_LAUNCHED(1);
    e = scan_exclusive_u32(keep, nA, idxA, cnt, st);
    if (e == cudaSuccess) {
      k_up_a<<<nblk(nA), 256, 0, st>>>(a, idxA, H, o, status);
      DMSC_LAUNCHED(1);
    }
  }
  if (e == cudaSuccess && nB) {
    k_up_b_classify<<<nblk(nB), 256, 0, st>>>(b, H, idxB, isnew);
    DMSC_LAUNCHED(1);
    e = scan_exclusive_u32(isnew, nB, posB, cnt + 1, st);
    if (e == cudaSuccess) {
      k_up_b_new<<<nblk(nB), 256, 0, st>>>(b, isnew, posB, cnt, H, idxB, o, status);
      DMSC_LAUNCHED(1);
    }
  }
  // boundary pairs (:84-92), A's then B's
  if (e == cudaSuccess && nA) { k_up_pairs<<<nblk(nA), 256, 0, st>>>(a, idxA, H, o.pair, status); DMSC_LAUNCHED(1); }
  if (e == cudaSuccess && nB) { k_up_pairs<<<nblk(nB), 256, 0, st>>>(b, idxB, H, o.pair, status); DMSC_LAUNCHED(1); }
  // connectivity (:94-121)
  if (e == cudaSuccess && nA) {
    k_up_count<<<nblk(nA), 256, 0, st>>>(a, idxA, false, ixn, tot_a, tot_d, mix, status);
    DMSC_LAUNCHED(1);
  }
  if (e == cudaSuccess && nB) {
    k_up_count<<<nblk(nB), 256, 0, st>>>(b, idxB, true, ixn, tot_a, tot_d, mix, status);
    DMSC_LAUNCHED(1);
  }
  if (e == cudaSuccess) e = scan_exclusive_u32(tot_a, bound, o.aoff, o.aoff + bound, st);
  if (e == cudaSuccess) e = scan_exclusive_u32(tot_d, bound, o.doff, o.doff + bound, st);
  if (e == cudaSuccess && nA) { k_up_write<<<nblk(nA), 256, 0, st>>>(a, idxA, false, ixn, o); DMSC_LAUNCHED(1); }
  if (e == cudaSuccess && nB) { k_up_write<<<nblk(nB), 256, 0, st>>>(b, idxB, true, ixn, o); DMSC_LAUNCHED(1); }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = sort_segments(bound, o.aoff, o.asc, mix, st);
  if (e == cudaSuccess) e = sort_segments(bound, o.doff, o.des, mix, st);
  uint32_t h[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, cnt, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h + 2, o.aoff + bound, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h + 3, o.doff + bound, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  s.free(st);
  if (e != cudaSuccess) return e;
  O.ncp = (long long)h[0] + h[1];
  O.nasc = h[2];
  O.ndes = h[3];
  O.any_bcancel = true;
  return cudaSuccess;
}

// A child's complex after merge_down, computed beside it (the child itself
// is replaced only once every merge of the level has succeeded).
struct ChildOut {
  DevBuf<uint32_t> cellid, pair_idx, aoff, asc, doff, des;
  DevBuf<float> fn;
  DevBuf<uint8_t> flags;
  long long ncp = 0, nasc = 0, ndes = 0;
};

template <typename T> void swap_buf(DevBuf<T> &a, DevBuf<T> &b) {
  std::swap(a.p, b.p);
  std::swap(a.n, b.n);
  std::swap(a.pooled, b.pooled);
}

void child_take(dmsc_msc &C, ChildOut &o, const int box[4]) {
  swap_buf(C.cellid, o.cellid); swap_buf(C.pair_idx, o.pair_idx); swap_buf(C.aoff, o.aoff); swap_buf(C.asc, o.asc);
  swap_buf(C.doff, o.doff); swap_buf(C.des, o.des); swap_buf(C.fn, o.fn); swap_buf(C.flags, o.flags);
  C.ncp = o.ncp; C.nasc = o.nasc; C.ndes = o.ndes;
  C.any_bcancel = true;
  for (int i = 0; i < 4; ++i) C.bbox[i] = box[i];
}

// merge_down of parent graph hp into child C (:207-320), into `out`.
// jb/njb: the parent's boundary-cancelable points; adds: a bound on the
// events (partners and list entries of those points); box: the child's box
// grown by the cells those points can add.
cudaError_t down_child(MGraphHost &hp, const uint32_t *jb, uint32_t njb, unsigned long long adds, const dmsc_msc &C,
                       const int box[4], ChildOut &out, uint32_t *status, cudaStream_t st) {
  const MGraph &P = mg(hp);
  const long long n0 = C.ncp, cap = n0 + (long long)adds + 1;
  if (cap >= (1ll << 31)) return cudaErrorInvalidValue;
  const int tw = box[2] - box[0] + 1, th = box[3] - box[1] + 1;
  if (tw <= 0 || th <= 0) return cudaErrorInvalidValue;
  const size_t cells = (size_t)tw * th;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = out.cellid.ensure(cap, st);
  if (e == cudaSuccess) e = out.fn.ensure(cap, st);
  if (e == cudaSuccess) e = out.pair_idx.ensure(cap, st);
  if (e == cudaSuccess) e = out.flags.ensure(cap, st);
  if (e == cudaSuccess) e = out.aoff.ensure(cap, st);
  if (e == cudaSuccess) e = out.doff.ensure(cap, st);
  if (e != cudaSuccess) return e;
  Scratch s;
  // tab, first, cnt, base, addsrc, kind, addf, rank, src, tot_a, tot_d, need, counters
  s.sz = {4 * cells, 4 * cells, 4ull * (njb + 1), 4ull * (njb + 1), 4ull * (njb + 1), (size_t)njb + 1,
          4ull * (adds + 1), 4ull * (adds + 1), 4ull * cap, 4ull * cap, 4ull * cap, (size_t)cap, 64};
  if ((e = s.alloc(st)) != cudaSuccess) return e;
  DcArgs a;
  a.P = P;
  a.jb = jb;
  a.njb = njb;
  a.c = csr_in(C);
  a.tab = CellTab{(uint32_t *)s.ptr[0], box[0], box[1], tw, th};
  a.first = CellTab{(uint32_t *)s.ptr[1], box[0], box[1], tw, th};
  a.cnt = (uint32_t *)s.ptr[2];
  a.base = (uint32_t *)s.ptr[3];
  a.addsrc = (uint32_t *)s.ptr[4];
  a.kind = (uint8_t *)s.ptr[5];
  a.addf = (uint32_t *)s.ptr[6];
  a.rank = (uint32_t *)s.ptr[7];
  uint32_t *src = (uint32_t *)s.ptr[8], *tot_a = (uint32_t *)s.ptr[9], *tot_d = (uint32_t *)s.ptr[10];
  uint8_t *need = (uint8_t *)s.ptr[11];
  uint32_t *ctr = (uint32_t *)s.ptr[12];  // [0] events, [1] added points
  a.o = CsrOut{out.cellid.p, out.pair_idx.p, out.aoff.p, nullptr, out.doff.p, nullptr, out.fn.p, out.flags.p};
  a.ncp0 = (uint32_t)n0;
  a.status = status;
  e = cudaMemsetAsync(s.ptr[0], 0xFF, 4 * cells, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(s.ptr[1], 0xFF, 4 * cells, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ctr, 0, 64, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(a.addf, 0, 4ull * (adds + 1), st);
  if (e == cudaSuccess && n0) {
    k_dc_table<<<nblk(n0), 256, 0, st>>>(a.c, a.tab, status);
    DMSC_LAUNCHED(1);
    e = cudaMemcpyAsync(out.cellid.p, C.cellid.p, 4ull * n0, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out.fn.p, C.fn.p, 4ull * n0, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out.pair_idx.p, C.pair_idx.p, 4ull * n0, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out.flags.p, C.flags.p, n0, cudaMemcpyDeviceToDevice, st);
  }
  if (e == cudaSuccess && njb) {
    k_dc_classify<<<nblk(njb), 256, 0, st>>>(a);
    DMSC_LAUNCHED(1);
    e = scan_exclusive_u32(a.cnt, njb, a.base, ctr, st);
    if (e == cudaSuccess) {
      k_dc_first<<<nblk(njb), 256, 0, st>>>(a);
      k_dc_addflags<<<nblk(njb), 256, 0, st>>>(a);
      DMSC_LAUNCHED(2);
      e = scan_exclusive_u32(a.addf, (long long)adds + 1, a.rank, ctr + 1, st);
    }
    if (e == cudaSuccess) {
      k_dc_add<<<nblk(njb), 256, 0, st>>>(a);
      k_dc_pairing<<<nblk(njb), 256, 0, st>>>(a);
      DMSC_LAUNCHED(2);
      e = cudaGetLastError();
    }
  }
  uint32_t hc[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(hc, ctr, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  const long long n = n0 + hc[1];
  if (e == cudaSuccess && (unsigned long long)hc[0] > adds) e = cudaErrorInvalidValue;  // the event bound failed
  // the lists (:283-320): taken from the parent where it holds the cell
  if (e == cudaSuccess && n) {
    k_dc_src<<<nblk(n), 256, 0, st>>>(a, (uint32_t)n, src);
    k_dc_count<<<nblk(n), 256, 0, st>>>(a, (uint32_t)n, src, tot_a, tot_d, need);
    DMSC_LAUNCHED(2);
  }
  if (e == cudaSuccess) e = scan_exclusive_u32(tot_a, n, out.aoff.p, out.aoff.p + n, st);
  if (e == cudaSuccess) e = scan_exclusive_u32(tot_d, n, out.doff.p, out.doff.p + n, st);
  uint32_t tot[2] = {0, 0};
  unsigned long long *sum = (unsigned long long *)(ctr + 4), hsum[2] = {0, 0};  // the same totals in 64 bits
  if (e == cudaSuccess) e = sum_u32(tot_a, n, sum, st);
  if (e == cudaSuccess) e = sum_u32(tot_d, n, sum + 1, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hsum, sum, 16, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[0], out.aoff.p + n, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[1], out.doff.p + n, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && std::max(hsum[0], hsum[1]) > 0xffffffffull) e = cudaErrorMemoryAllocation;  // 32-bit offsets
  if (e == cudaSuccess) e = out.asc.ensure((size_t)tot[0] + 1, st);
  if (e == cudaSuccess) e = out.des.ensure((size_t)tot[1] + 1, st);
  if (e == cudaSuccess && n) {
    a.o.asc = out.asc.p;
    a.o.des = out.des.p;
    k_dc_write<<<nblk(n), 256, 0, st>>>(a, (uint32_t)n, src);
    DMSC_LAUNCHED(1);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = sort_segments(n, out.aoff.p, out.asc.p, need, st);
  if (e == cudaSuccess) e = sort_segments(n, out.doff.p, out.des.p, need, st);
  s.free(st);
  if (e != cudaSuccess) return e;
  out.ncp = n;
  out.nasc = tot[0];
  out.ndes = tot[1];
  return cudaSuccess;
}

}  // namespace

namespace {
constexpr int MERGE_WORKERS = 8;

cudaError_t as_cuda(int rc) {
  return rc == 0 ? cudaSuccess : rc < 0 ? cudaErrorUnknown : (cudaError_t)rc;
}
int current_device() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}
}  // namespace

// The merges of a level run side by side on their own streams (several host
// threads); the boundary steps of all of them run in one launch on `st`.
cudaError_t merge_up_level_par(const std::vector<MergeJob> &jobs, unsigned long long grow, uint32_t *status,
                               uint32_t *stw, cudaStream_t st, double *seq_ms, long long round_window,
                               long long round_min_commits) {
  *stw = 0;
  const int nj = (int)jobs.size(), dev = current_device();
  cudaError_t e = cudaMemsetAsync(status, 0, 4, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  // union and connectivity; each result's cell table passes to its graph
  std::vector<MGraphHost> g(nj);
  std::vector<uint32_t *> tabs(nj, nullptr);
  if (e == cudaSuccess)
    e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS, [&](int k, cudaStream_t s) {
      const MergeJob &J = jobs[k];
      return (int)union_one(*J.a, *J.b, *J.parent, CRect{J.ixn[0], J.ixn[1], J.ixn[2], J.ixn[3]}, status, &tabs[k], s);
    }));
  if (e == cudaSuccess) e = cudaMemcpy(stw, status, 4, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess || *stw) {
    for (uint32_t *t : tabs)
      if (t) cudaFreeAsync(t, st);
    cudaStreamSynchronize(st);
    return e;
  }
  // the boundary cancellations, up to UP_BLOCKS blocks per merge, on mutable graphs
  std::vector<MGraphHost *> gp;
  std::vector<SeqJob> seq;
  for (int k = 0; k < nj; ++k) {
    const int *x = jobs[k].ixn;
    gp.push_back(&g[k]);
    SeqJob j{SEQ_UP_CANCEL, k, CRect{x[0], x[1], x[2], x[3]}};
    j.win = (int)std::min<long long>(std::max<long long>(round_window, 0), 1 << 30);
    j.min_commits = (int)std::min<long long>(std::max<long long>(round_min_commits, 0), 1 << 30);
    seq.push_back(j);
  }
  e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS, [&](int k, cudaStream_t s) {
    const dmsc_msc &O = *jobs[k].parent;
    g[k].status = status;
    const cudaError_t r =
        mgraph_alloc(g[k], O, (uint32_t)O.ncp, O.nasc + O.ndes + grow * boundary_room(jobs[k].ixn), s, 0, tabs[k]);
    if (g[k].tab) tabs[k] = nullptr;  // the graph owns it now
    return (int)r;
  }));
  for (uint32_t *t : tabs)
    if (t) cudaFreeAsync(t, st);
  if (e == cudaSuccess) e = run_seq(gp, seq, status, st, seq_ms);
  if (e == cudaSuccess) e = cudaMemcpy(stw, status, 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && !*stw)
    e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS,
                                    [&](int k, cudaStream_t s) { return (int)mgraph_to_csr(g[k], *jobs[k].parent, s); }));
  for (auto &h : g) mgraph_free(h, st);
  cudaStreamSynchronize(st);
  return e;
}

cudaError_t merge_down_level_par(const std::vector<MergeJob> &jobs, unsigned long long grow, uint32_t *status,
                                 uint32_t *stw, cudaStream_t st, double *seq_ms) {
  *stw = 0;
  const int nj = (int)jobs.size(), dev = current_device();
  cudaError_t e = cudaMemsetAsync(status, 0, 4, st);
  // the parents' graphs
  std::vector<MGraphHost> g(nj);
  std::vector<MGraphHost *> gp;
  for (auto &h : g) gp.push_back(&h);
  std::vector<SeqJob> seq;
  for (int k = 0; k < nj; ++k) {
    const int *x = jobs[k].ixn;
    seq.push_back(SeqJob{SEQ_DOWN_BOUNDARY, k, CRect{x[0], x[1], x[2], x[3]}});
  }
  // scratch: per job the boundary-cancelable flags, positions and list; counters
  Scratch s;
  for (int k = 0; k < nj; ++k) {
    const long long n = jobs[k].parent->ncp;
    for (int q = 0; q < 3; ++q) s.sz.push_back(4ull * (n + 1));
  }
  s.sz.push_back(16ull * (nj + 1));  // per job: count, adds
  s.sz.push_back(16ull * (nj + 1));  // per job: the box of the cells its boundary points can add
  if (e == cudaSuccess) e = s.alloc(st);
  unsigned long long *ctr = e == cudaSuccess ? (unsigned long long *)s.ptr[3 * nj] : nullptr;
  int *boxes = e == cudaSuccess ? (int *)s.ptr[3 * nj + 1] : nullptr;
  std::vector<int> hbox(4 * (nj + 1));
  for (int k = 0; k <= nj; ++k) {
    hbox[4 * k] = hbox[4 * k + 1] = 1 << 30;
    hbox[4 * k + 2] = hbox[4 * k + 3] = -1;
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(ctr, 0, 16ull * (nj + 1), st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(boxes, hbox.data(), 16ull * (nj + 1), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess)
    e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS, [&](int k, cudaStream_t q) {
      const dmsc_msc &P = *jobs[k].parent;
      g[k].status = status;
      return (int)mgraph_alloc(g[k], P, (uint32_t)P.ncp, P.nasc + P.ndes + grow * boundary_room(jobs[k].ixn), q, 0);
    }));
  // the uncancellations along each shared boundary (:172-201)
  if (e == cudaSuccess) e = run_seq(gp, seq, status, st, seq_ms);
  // checks, the boundary-cancelable lists and the bounds of the children's growth
  if (e == cudaSuccess)
    e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS, [&](int k, cudaStream_t q) {
      MGraph &P = mg(g[k]);
      uint32_t *bflag = (uint32_t *)s.ptr[3 * k], *pos = (uint32_t *)s.ptr[3 * k + 1], *jb = (uint32_t *)s.ptr[3 * k + 2];
      uint32_t *njb = (uint32_t *)(ctr + 2 * k);
      if (!P.G.ncp) return 0;
      k_down_check<<<nblk(P.G.ncp), 256, 0, q>>>(P, bflag, status);
      DMSC_LAUNCHED(1);
      cudaError_t r = scan_exclusive_u32(bflag, P.G.ncp, pos, njb, q);
      if (r == cudaSuccess) {
        k_down_list<<<nblk(P.G.ncp), 256, 0, q>>>(P, bflag, pos, jb, ctr + 2 * k + 1, boxes + 4 * k);
        DMSC_LAUNCHED(1);
        r = cudaGetLastError();
      }
      return (int)r;
    }));
  std::vector<unsigned long long> hc(2 * (nj + 1), 0);
  if (e == cudaSuccess) e = cudaMemcpy(hc.data(), ctr, 16ull * nj, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(hbox.data(), boxes, 16ull * nj, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(stw, status, 4, cudaMemcpyDeviceToHost);
  // each child's box grows by the cells its parent's boundary points can add
  std::vector<int> cbox(8 * nj);
  for (int k = 0; k < nj; ++k)
    for (int c = 0; c < 2; ++c) {
      const dmsc_msc &C = *(c ? jobs[k].b : jobs[k].a);
      int *o = &cbox[8 * k + 4 * c];
      const int *t = &hbox[4 * k];
      for (int i = 0; i < 4; ++i) o[i] = C.bbox[i];
      if (t[2] >= 0) {
        o[0] = std::min(o[0], t[0]); o[1] = std::min(o[1], t[1]);
        o[2] = std::max(o[2], t[2]); o[3] = std::max(o[3], t[3]);
      }
    }
  // the parent into each child (:207-320), beside the child
  std::vector<ChildOut> outs(2 * nj);
  if (e == cudaSuccess && !*stw)
    e = as_cuda(for_each_on_streams(dev, 2 * nj, MERGE_WORKERS, [&](int kc, cudaStream_t q) {
      const int k = kc / 2, c = kc % 2;
      const dmsc_msc &C = *(c ? jobs[k].b : jobs[k].a);
      return (int)down_child(g[k], (const uint32_t *)s.ptr[3 * k + 2], (uint32_t)hc[2 * k], hc[2 * k + 1], C,
                             &cbox[8 * k + 4 * c], outs[kc], status, q);
    }));
  if (e == cudaSuccess && !*stw) e = cudaMemcpy(stw, status, 4, cudaMemcpyDeviceToHost);
  // every merge of the level succeeded: the children take their new
  // complexes and the parents are written back
  if (e == cudaSuccess && !*stw) {
    for (int kc = 0; kc < 2 * nj; ++kc) child_take(*(kc % 2 ? jobs[kc / 2].b : jobs[kc / 2].a), outs[kc], &cbox[4 * kc]);
    e = as_cuda(for_each_on_streams(dev, nj, MERGE_WORKERS,
                                    [&](int k, cudaStream_t q) { return (int)mgraph_to_csr(g[k], *jobs[k].parent, q); }));
  }
  s.free(st);
  for (auto &h : g) mgraph_free(h, st);
  cudaStreamSynchronize(st);
  return e;
}

}  // namespace dmsc
