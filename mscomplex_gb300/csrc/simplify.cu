// simplify.cu -- persistence simplification of a Morse-Smale complex on the
// device: GridMSComplex::simplify + un_simplify (dmsc/src/grid_mscomplex.cpp:
// 384-526) with cancelPairs (dmsc/include/discreteMorseAlgorithm.h:466-585)
// and uncancel_pairs (:1006-1089).
//
// The reference pops a std::priority_queue whose comparator (grid_mscomplex.cpp:
// 331-379) reads c3/c4 from p1, so for equal persistence it returns false both
// ways: the order among ties is whatever the binary-heap algorithms produce.
// The result depends on that order (including the order produced by the
// strangulation resubmissions, :474-479, 503-508), so this pass replays the
// heap exactly: the standard bottom-up binary heap of push_heap / pop_heap
// (hole sifted down to a leaf choosing the right child unless the left one is
// strictly smaller, then the last element sifted up) -- the algorithm of the
// C++ standard library the reference is built with.  Persistence |f2 - f1| is
// precomputed per heap entry; the comparator is "d1 > d2" (a min-heap on d).
//
// The replay is sequential by nature: one warp of one block makes the heap
// operations and graph edits in order, and its lanes share the work inside
// each of them (struct Simp; warp_graph.cuh).  Multisets
// (critical_point::asc / des, std::multiset<uint>) are run-length encoded
// sorted arrays in a device pool; they grow by reallocation inside it.  Every
// loop is bounded: the pass stops with ST_SIMPLIFY_LIMIT when the operation
// budget or a pool runs out, leaving the complex unmodified.
#include "dmsc_common.cuh"
#include "dmsc_internal.h"
#include "msc_graph.cuh"
#include "smem_limit.h"
#include "warp_graph.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace dmsc {

// A heap entry: persistence and the pair (a, b).  The top three bits of a
// and of b carry that critical point's static facts (on rect's boundary, cell
// dimension), so that a popped pair is classified from the entry itself and
// a resubmitted pair goes back on the heap without a load.  Critical point
// indices are below 2^29.
struct HeapEnt {
  float d;
  uint32_t a, b;
};
constexpr uint32_t IDX_MASK = (1u << 29) - 1u, META_BOUNDARY = 1u << 31;
__host__ __device__ __forceinline__ uint32_t ent_idx(uint32_t x) { return x & IDX_MASK; }
__host__ __device__ __forceinline__ int ent_dim(uint32_t x) { return (int)((x >> 29) & 3u); }
__host__ __device__ __forceinline__ bool ent_boundary(uint32_t x) { return (x & META_BOUNDARY) != 0; }

// IEEE single subtraction without contraction on either side of the compiler.
__host__ __device__ __forceinline__ float fsub_rn(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  volatile float r = a - b;
  return r;
#endif
}

__host__ __device__ __forceinline__ float bits_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, 4);
  return f;
#endif
}
__host__ __device__ __forceinline__ uint32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u;
#endif
}
// The loop stops at the first pair with (double)d / (double)max_persistence >
// tresh (grid_mscomplex.cpp:446-447).  A correctly rounded division by a
// fixed divisor is monotone in d, so over the persistences (non-negative,
// finite floats, whose bit patterns order like their values) the test is
// true exactly from one bit pattern on.  That pattern is found once here, by
// bisection with the same double-precision test, and each pop compares bits:
// the same outcome for every d, without a double division per pop (double
// precision is slow on this part).  Returns 0x7F800001 if no finite d passes.
__host__ __device__ inline uint32_t stop_bits(float max_persistence, double tresh) {
  auto over = [&](uint32_t u) { return (double)bits_float(u) / (double)max_persistence > tresh; };
  uint32_t lo = 0, hi = 0x7F800001u;  // the first passing pattern lies in [lo, hi]
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (over(mid)) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

struct SimpArgs {
  Graph G;            // the complex as a mutable graph (msc_graph.cuh)
  const float *fn;
  uint32_t *meta;     // per critical point: its index with the entry bits (k_simp_meta); its pair's order (k_unsimplify)
  float *hkey;        // the heap in global memory, keys and pairs apart, entries 1 .. heap_cap
  uint2 *hab;
  unsigned long long heap_cap;
  HeapEnt *resub;     // resubmit list (capacity heap_cap), whole entries
  uint2 *canc;        // cancellation list (capacity ncp)
  uint32_t ncanc;     // its length, and whether it holds a pair that was not connected (for k_unsimplify)
  bool loose;
  int rx0, ry0, rx1, ry1;  // m_rect of the complex (cell coordinates)
  double tresh;
  unsigned long long *stats;  // [0] pushes [1] pops [2] cancels [3] ops [4] status [5] asc [6] des entries
  // the complex's CSR lists (offsets may be based anywhere) and the entries of
  // its first pushes, one per des arc in that order (k_simp_prep)
  const uint32_t *aoff, *asc, *doff, *des;
  HeapEnt *init;
  unsigned long long ninit;
};

// The heap's first TL levels, which every pop walks, live in shared memory,
// the rest in global memory; both hold keys and (a, b) pairs in separate
// arrays indexed from 1 (entry k has the children 2k and 2k + 1), so that one
// aligned 8-byte load gets both children's keys.
constexpr int TOP_LEVELS = 14, TOP_LEVELS_BATCH = 13;
// The block's warps: the first replays the heap, the others edit the lists
// of cancelled pairs, each with shared memory for a long list's edit.
constexpr int SIMP_WARPS = 4, HELPERS = SIMP_WARPS - 1;
__host__ __device__ constexpr uint32_t edit_runs(int levels) { return levels == TOP_LEVELS ? 1024 : 512; }
__host__ __device__ constexpr size_t top_bytes(int levels) {
  return ((sizeof(float) + sizeof(uint2)) << levels) + sizeof(uint2) * HELPERS * edit_runs(levels);
}
// The state the warps share: the pair being cancelled, and whether to stop.
// The first warp starts the helpers through barrier BAR_GO and waits for them
// through BAR_DONE; each is passed by every thread of the block once per
// cancellation (BAR_GO once more at the end, with stop set).
struct SimpShared {
  TeamState team;
  WarpGraph::Pair pair;
  int stop;
};
constexpr int BAR_GO = 1, BAR_DONE = 2;
__device__ __forceinline__ void bar_arrive(int b) {
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"r"(b), "r"(32 * SIMP_WARPS) : "memory");
}
__device__ __forceinline__ void bar_wait(int b) {
  asm volatile("bar.sync %0, %1;" ::"r"(b), "r"(32 * SIMP_WARPS) : "memory");
}
constexpr unsigned long long HEAP_MAX = 0xFFFFFFE0ull;  // entries: 32-bit indices, one lane per level in a push

// The replay by one warp.  What bounds it is the latency of each dependent
// step, so the lanes take the steps of one heap operation together:
//   * pop: the hole's path to the leaves depends on the keys alone.  Each lane
//     compares the two children of one node of the 5-level subtree under the
//     hole; a ballot of the choices tells every lane whether its node lies on
//     the path (its ancestors' choices, a mask of constants per lane), so one
//     load and two ballots replace five dependent loads, and the path's entries
//     move up together;
//   * push: one lane per ancestor compares its key; a ballot gives the climb;
//   * a burst of pushes (the first pushes, the resubmit list, new edges): 32
//     at a time, the entries that stay where they are pushed (their parent is
//     not larger) are stored at once.
// A cancellation's list edits go to the block's other warps (help): they are
// chains of dependent loads of lists no one has touched for long, and until
// the next pair is classified the heap needs none of them, so they run beside
// the pushes of the new edges and of the resubmit list and the next pop.
// On the 256x256 noisy field at 5% (35,000 pops, 1,520 cancellations) one
// thread took 2,150 cycles a pop, 710 a push and 23,000 a cancellation, 74 ms
// in all; here a pop takes 750, a push 225 and a cancellation waits 550 for
// its edits, 24 ms in all.
struct Simp {
  SimpArgs A;
  WarpGraph W;
  float *skey;
  uint2 *sab;
  uint32_t ntop;                  // entries below it are in shared memory (a power of two)
  uint32_t nheap = 0, nres = 0, ncanc = 0;
  unsigned long long n_pop = 0;   // heap operations (the pushes: the pops and what is left)
  bool ordered = false;           // no key is NaN (all values finite)
  bool loose = false;             // a pair that was not connected is on the cancellation list
  // this lane's node of the 5-level subtree under entry h is h * mul + add (lane 31: none), its
  // ancestors among the lanes are anc, and those of them in need must choose the right child
  uint32_t mul, add, anc, need;

  SimpShared *sh;
  bool pending = false;           // the helpers are at work

  __device__ Simp(const SimpArgs &a, void *smem, int levels, SimpShared *shared) : A(a), sh(shared) {
    W.G = a.G;
    W.lane = threadIdx.x & 31;
    ntop = 1u << levels;
    sab = reinterpret_cast<uint2 *>(smem);
    skey = reinterpret_cast<float *>(sab + ntop);
    const uint32_t i = (uint32_t)W.lane + 1;  // 1-based node of the subtree
    const int ll = 31 - __clz(i);
    mul = 1u << ll;
    add = i - mul;
    anc = need = 0;
    for (int s = 1; s <= ll; ++s) {
      anc |= 1u << ((i >> s) - 1);
      if ((i >> (s - 1)) & 1u) need |= 1u << ((i >> s) - 1);
    }
    if (W.lane == 31) { mul = 0; add = 0xFFFFFFFFu; }
    W.stage = nullptr;
    W.nstage = 0;
  }
  // waits for the helpers' edits
  __device__ __forceinline__ void settle() {
    if (!pending) return;
    pending = false;
    bar_wait(BAR_DONE);
    if (sh->team.fail) W.G.fail = true;
    W.G.ops += sh->team.ops;
    __syncwarp();
    if (W.lane == 0) sh->team.ops = 0;
    __syncwarp();
  }
  __device__ __forceinline__ float key_at(uint32_t k) const { return k < ntop ? skey[k] : A.hkey[k]; }
  __device__ __forceinline__ void put(uint32_t k, float d, uint2 ab) {
    if (k < ntop) { skey[k] = d; sab[k] = ab; }
    else { A.hkey[k] = d; A.hab[k] = ab; }
  }

  // __push_heap from entry k (comparator d1 > d2): the entry climbs while its
  // parent is larger.  Lane l holds the ancestor l + 1 levels up and, where
  // every lane below it climbs, fills the place l levels up.
  template <bool TOP>  // TOP: entry k, and so all of its ancestors, in shared memory
  __device__ __forceinline__ void push_at(uint32_t k, float d, uint2 ab) {
    const uint32_t to = k >> W.lane, p = to >> 1;
    float pk;
    uint2 pab;
    if (TOP || p < ntop) {  // (entry 0 is never used)
      pk = skey[p];
      pab = sab[p];
    } else {
      pk = A.hkey[p];
      pab = A.hab[p];
    }
    const bool climbs = p != 0 && pk > d;
    const unsigned up = __ballot_sync(FULL_WARP, climbs);
    if ((~up & W.lt()) == 0) {
      pk = climbs ? pk : d;
      pab = climbs ? pab : ab;
      if (TOP) { skey[to] = pk; sab[to] = pab; }
      else put(to, pk, pab);
    }
    __syncwarp();
  }
  // The lanes of `mask` push their entries, in lane order.  An entry whose
  // parent is not larger stays at its own place and changes no other; the
  // climbs of the others only lower the keys of their ancestors (where the
  // keys are ordered), so it stays there whether they come before or after it.
  template <bool TOP>
  __device__ __forceinline__ void push_lanes_t(unsigned mask, uint32_t cnt, float d, uint2 ab) {
    const uint32_t k = nheap + 1 + __popc(mask & W.lt());
    unsigned todo = mask;
    if (ordered && nheap >= 32) {  // every parent is an older entry
      const bool on = (mask >> W.lane) & 1u;
      const uint32_t p = on ? k >> 1 : 0;
      const bool climbs = on && (TOP ? skey[p] : key_at(p)) > d;
      if (on && !climbs) {
        if (TOP) { skey[k] = d; sab[k] = ab; }
        else put(k, d, ab);
      }
      todo = __ballot_sync(FULL_WARP, climbs);
    }
    nheap += cnt;
    // the next entry is on its way while one climbs
    uint32_t nk = 0;
    float ndv = 0.0f;
    uint2 nab = make_uint2(0, 0);
    auto next = [&]() {
      const int s = (__ffs(todo) - 1) & 31;
      nk = __shfl_sync(FULL_WARP, k, s);
      ndv = __shfl_sync(FULL_WARP, d, s);
      nab = make_uint2(__shfl_sync(FULL_WARP, ab.x, s), __shfl_sync(FULL_WARP, ab.y, s));
    };
    next();
    while (todo) {
      const uint32_t ck = nk;
      const float cd = ndv;
      const uint2 cab = nab;
      todo &= todo - 1;
      next();
      push_at<TOP>(ck, cd, cab);
    }
  }
  __device__ __forceinline__ void push_lanes(unsigned mask, float d, uint2 ab) {
    __syncwarp();
    const uint32_t cnt = __popc(mask);
    if ((unsigned long long)nheap + cnt > A.heap_cap) { W.G.fail = true; return; }
    if (nheap + cnt < ntop) push_lanes_t<true>(mask, cnt, d, ab);
    else push_lanes_t<false>(mask, cnt, d, ab);
  }
  __device__ __forceinline__ static unsigned first_lanes(unsigned long long n) {
    return n >= 32 ? FULL_WARP : (1u << (unsigned)n) - 1u;
  }
  __device__ __forceinline__ void push_entries(const HeapEnt *src, unsigned long long n) {
    __syncwarp();
    HeapEnt nx{0.0f, 0, 0};
    if ((unsigned)W.lane < n) nx = src[W.lane];
    for (unsigned long long q = 0; q < n && !W.G.fail; q += 32) {
      const HeapEnt e = nx;
      if (q + 32 + W.lane < n) nx = src[q + 32 + W.lane];  // the next 32 on their way
      push_lanes(first_lanes(n - q), e.d, make_uint2(e.a, e.b));
    }
  }
  // pushes (d, a) for every occurrence of a value in p[0..n) but `skip`, in
  // order: the value is the pair's second point with `other` the first
  // (second = true), or the other way round
  __device__ __forceinline__ void push_edges(const uint2 *p, uint32_t n, uint32_t skip, uint32_t other, bool second) {
    const float fo = A.fn[other];
    const uint32_t mo = A.meta[other];
    for (uint32_t i0 = 0; i0 < n && !W.G.fail; i0 += 32) {
      uint2 r = make_uint2(skip, 0);
      if (i0 + W.lane < n) r = p[i0 + W.lane];
      const bool on = r.x != skip;
      const uint32_t at = on ? r.x : other;
      const uint32_t mr = A.meta[at];
      const float fr = A.fn[at];
      const float d = fabsf(second ? fsub_rn(fr, fo) : fsub_rn(fo, fr));
      const uint2 ab = second ? make_uint2(mo, mr) : make_uint2(mr, mo);
      const unsigned many = __ballot_sync(FULL_WARP, on && r.y > 1), all = __ballot_sync(FULL_WARP, on);
      if (!many) {
        push_lanes(all, d, ab);
        continue;
      }
      for (unsigned todo = all; todo && !W.G.fail; todo &= todo - 1) {  // copies: one value after the other
        const int s = __ffs(todo) - 1;
        const uint32_t c = __shfl_sync(FULL_WARP, r.y, s);
        const float ds = __shfl_sync(FULL_WARP, d, s);
        const uint2 as = make_uint2(__shfl_sync(FULL_WARP, ab.x, s), __shfl_sync(FULL_WARP, ab.y, s));
        for (uint32_t q = 0; q < c && !W.G.fail; q += 32) push_lanes(first_lanes(c - q), ds, as);
      }
    }
  }

  // pop_heap + pop_back: libstdc++'s __adjust_heap moves the hole from the
  // root to a leaf along the smaller children (the right one unless the left
  // is strictly smaller), then sifts the last element up from that leaf.  The
  // sift-up restores every path entry below the place where the last element
  // lands, so the hole stops there -- at the first chosen child larger than
  // the last element -- which leaves the same heap with fewer moves.  The
  // popped entry is on top before the call.
  __device__ __forceinline__ void pop() {
    ++n_pop;
    if (nheap < ntop) pop_t<true>();
    else pop_t<false>();
  }
  template <bool TOP>  // TOP: the whole heap in shared memory
  __device__ __forceinline__ void pop_t() {
    const uint32_t last = nheap, len = --nheap;  // entries 1 .. len remain
    if (len == 0) return;
    float vd;
    uint2 vab;
    if (TOP) {
      vd = skey[last];
      vab = sab[last];
    } else {
      vd = A.hkey[last];
      vab = A.hab[last];
      // the next pops' last elements: their lines on their way into L1
      if (len >= ntop + 32) {
        if (W.lane == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(A.hkey + len - 32));
        if (W.lane == 1) asm volatile("prefetch.global.L1 [%0];" ::"l"(A.hab + len - 16));
      }
    }
    // shared-memory levels: the path from the keys alone, five levels a round
    constexpr int R = 3;
    const uint32_t lim = TOP ? len : ntop - 1;
    const uint32_t half = lim >> 1, half1 = (lim - 1) >> 1;  // the last entries with a left / a right child there
    float ck[R];
    uint32_t nd[R], h = 1;
    uint2 mv[R];
    bool on[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      on[r] = false;
      nd[r] = 0;
      ck[r] = 0.0f;
      if (lim >= (2u << (5 * r))) {  // (known early: the path's own end is found without branches)
        nd[r] = h * mul + add;
        const bool has = nd[r] <= half;
        float2 kk = make_float2(0.0f, 0.0f);
        if (has) kk = reinterpret_cast<const float2 *>(skey)[nd[r]];
        const bool right = nd[r] <= half1 && !(kk.y > kk.x);
        const unsigned D = __ballot_sync(FULL_WARP, right);
        on[r] = has && ((D ^ need) & anc) == 0;
        const uint32_t child = 2 * nd[r] + (right ? 1u : 0u);
        ck[r] = right ? kk.y : kk.x;
        if (on[r]) mv[r] = sab[child];
        h = __reduce_max_sync(FULL_WARP, on[r] ? child : h);  // the path's last child
      }
    }
    // the first path node whose chosen child is larger than the last element;
    // the entries above it move up
    uint32_t place = 0xFFFFFFFFu;
#pragma unroll
    for (int r = R - 1; r >= 0; --r)
      if (on[r] && ck[r] > vd) place = nd[r];
    place = __reduce_min_sync(FULL_WARP, place);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (on[r] && nd[r] < place) { skey[nd[r]] = ck[r]; sab[nd[r]] = mv[r]; }
    __syncwarp();
    if (TOP) {  // (every lane stores the same)
      place = place == 0xFFFFFFFFu ? h : place;
      skey[place] = vd;
      sab[place] = vab;
    } else {
      if (place == 0xFFFFFFFFu) place = pop_global(h, len, vd);
      if (W.lane == 0) put(place, vd, vab);
    }
    __syncwarp();
  }
  // the levels in global memory, five a round trip; the place of the last element
  __device__ __forceinline__ uint32_t pop_global(uint32_t h, uint32_t len, float vd) {
    const uint32_t half = len >> 1, half1 = (len - 1) >> 1;
    while (h <= half) {
      const unsigned long long nd = (unsigned long long)h * mul + add;
      const bool has = nd <= half;
      float2 kk = make_float2(0.0f, 0.0f);
      if (has) kk = reinterpret_cast<const float2 *>(A.hkey)[nd];
      const bool right = nd <= half1 && !(kk.y > kk.x);
      const unsigned D = __ballot_sync(FULL_WARP, right);
      bool on = has && ((D ^ need) & anc) == 0;
      const uint32_t child = 2 * (uint32_t)nd + (right ? 1u : 0u);
      const float ck = right ? kk.y : kk.x;
      const uint32_t place = __reduce_min_sync(FULL_WARP, on && ck > vd ? (uint32_t)nd : 0xFFFFFFFFu);
      h = __reduce_max_sync(FULL_WARP, on ? child : 0u);
      on = on && nd < place;
      uint2 mv;
      if (on) mv = A.hab[child];
      __syncwarp();
      if (on) put((uint32_t)nd, ck, mv);
      __syncwarp();
      if (place != 0xFFFFFFFFu) return place;
    }
    return h;
  }

  // simplify (grid_mscomplex.cpp:384-512)
  __device__ __forceinline__ void run() {
    Graph &G = W.G;
    const uint32_t n = G.ncp;
    const bool lead = W.lane == 0;
    // (:396-428) the strangulation marks and the entries of the first pushes
    // come from k_simp_prep; the value range and the pushes, in the
    // reference's order, here
    float max_val = 1.17549435e-38f;  // std::numeric_limits<float>::min(), as in the reference (:399)
    float min_val = 3.40282347e+38f;
    for (uint32_t i = W.lane; i < n; i += 32) {
      const float f = A.fn[i];
      max_val = (max_val < f) ? f : max_val;  // std::max
      min_val = (f < min_val) ? f : min_val;  // std::min
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float a = __shfl_xor_sync(FULL_WARP, max_val, o), b = __shfl_xor_sync(FULL_WARP, min_val, o);
      max_val = (max_val < a) ? a : max_val;
      min_val = (b < min_val) ? b : min_val;
    }
    ordered = max_val <= 3.40282347e+38f && min_val >= -3.40282347e+38f;
    push_entries(A.init, A.ninit);
    if (G.fail) nheap = 0;  // (nothing is popped; the pass has failed)
    const float max_persistence = fsub_rn(max_val, min_val);
    const uint32_t stop_at = stop_bits(max_persistence, A.tresh);
    const uint32_t ncl = n ? n - 1 : 0;
    float rd = 0.0f;  // resubmitted entries past the last full 32, one per lane
    uint2 rab = make_uint2(0, 0);
    while (nheap != 0) {
      ++G.ops;
      // the entry on top and its pair's dynamic state (three independent
      // loads), issued before the pop's descent so that they arrive during it
      const float ed = skey[1];
      const uint2 eab = sab[1];
      const bool turn = ent_dim(eab.y) == 1;
      const uint32_t w1 = turn ? eab.y : eab.x, w2 = turn ? eab.x : eab.y;
      const uint32_t v1 = ent_idx(w1), v2 = ent_idx(w2);
      const int cp2_dim = ent_dim(w2);
      const uint32_t u1 = min(v1, ncl), u2 = min(v2, ncl);
      uint32_t f1 = 0, f2 = 0, tot2 = 0;
      uint2 dsc = make_uint2(0, 0);
      auto state = [&]() {
        f1 = G.flags[u1];
        f2 = G.flags[u2];
        tot2 = G.L.total[2 * u2 + cp2_dim / 2];
        // should the pair be cancelled: its lists' places and lengths, one word pair per lane
        dsc = reinterpret_cast<const uint2 *>((W.lane & 1) ? G.L.nrun : G.L.off)[(W.lane & 2) ? u2 : u1];
      };
      if (!pending) state();
      __syncwarp();  // every lane has read the top
      pop();
      if (pending) {
        settle();
        if (G.fail) break;
        state();
      }
      const bool b1 = ent_boundary(w1), b2 = ent_boundary(w2), strang = f1 & F_STRANG;
      const bool stop = G.ops > G.max_ops || float_bits(ed) >= stop_at;  // (double)d / max_persistence > tresh
      const bool inside = v1 == u1 && v2 == u2;
      const bool skip = ((f1 | f2) & F_CANCELLED) || b1 != b2;
      const bool again = strang && tot2 != 1;
      if (!stop && inside && (skip || again)) {  // most pops
        const bool mine = !skip && (uint32_t)W.lane == (nres & 31u);
        rd = mine ? ed : rd;
        rab = mine ? eab : rab;
        nres += skip ? 0u : 1u;
        if (!skip && (nres & 31u) == 0) {
          if (nres > A.heap_cap) { G.fail = true; break; }
          A.resub[nres - 32 + W.lane] = HeapEnt{rd, rab.x, rab.y};
        }
        continue;
      }
      if (stop) {
        if (G.ops > G.max_ops) {  // the budget ends before this pop
          G.fail = true;
          --n_pop;
          ++nheap;
        }
        break;
      }
      if (!inside) {  // a list entry outside the complex
        if (lead) A.stats[4] |= ST_INVARIANT;
        continue;
      }
      if (strang && b1) continue;
      // (an asc list holds points of the next dimension only)
      uint2 pl[2], nr[2];  // of v1, v2
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        pl[q] = make_uint2(__shfl_sync(FULL_WARP, dsc.x, 2 * q), __shfl_sync(FULL_WARP, dsc.y, 2 * q));
        nr[q] = make_uint2(__shfl_sync(FULL_WARP, dsc.x, 2 * q + 1), __shfl_sync(FULL_WARP, dsc.y, 2 * q + 1));
      }
      WarpGraph::Pair pr = cp2_dim == 0 ? WarpGraph::Pair{pl[1], pl[0], nr[1], nr[0], v2, v1}
                                        : WarpGraph::Pair{pl[0], pl[1], nr[0], nr[1], v1, v2};
      const bool connected = W.orient(pr);
      if (ncanc >= n) { G.fail = true; break; }
      if (lead) {
        if (connected) sh->pair = pr;
        G.pair_idx[v1] = v2;
        G.pair_idx[v2] = v1;
        A.canc[ncanc] = connected ? make_uint2(pr.cp0, pr.cp1) : make_uint2(ent_idx(eab.x), ent_idx(eab.y));
        if (!connected) {
          G.flags[v1] |= F_BCANCEL;
          G.flags[v2] |= F_BCANCEL;
        }
      }
      ++ncanc;
      loose |= !connected;
      if (connected) {
        W.close(pr, F_BCANCEL);
        __syncwarp();
        bar_arrive(BAR_GO);
        pending = true;
      }
      __syncwarp();
      if (connected) {  // new edges (d, a), a in asc(cp0) \ {cp1}, d in des(cp1) \ {cp0}, in the reference's order
        const uint32_t cp0 = pr.cp0, cp1 = pr.cp1, na = pr.n0.x, nd = pr.n1.y;
        const uint2 *pa = G.L.pool + pr.o0.x, *pd = G.L.pool + pr.o1.y;
        uint2 r0 = make_uint2(cp0, 0), r1 = r0;  // des(cp1), when short
        if (nd > 0) r0 = pd[0];
        if (nd > 1) r1 = pd[1];
        const uint2 one = r0.x != cp0 ? r0 : r1;
        if (nd <= 2 && (r0.x == cp0 || r1.x == cp0) && (one.x == cp0 || one.y == 1)) {  // one d, or none
          if (one.x != cp0) push_edges(pa, na, cp1, one.x, true);
        } else {
          for (uint32_t i = 0; i < na && !G.fail; ++i) {
            const uint2 ra = pa[i];
            if (ra.x == cp1) continue;
            for (uint32_t ca = 0; ca < ra.y && !G.fail; ++ca) push_edges(pd, nd, cp0, ra.x, false);
          }
        }
      }
      if (!G.fail) {
        push_entries(A.resub, nres & ~31u);
        if (!G.fail && (nres & 31u)) push_lanes(first_lanes(nres & 31u), rd, rab);
      }
      if (G.fail) break;
      nres = 0;
    }
    settle();
    if (G.ops > G.max_ops) G.fail = true;
    if (lead) {
      A.stats[0] = n_pop + nheap;
      A.stats[1] = n_pop;
      A.stats[2] = ncanc;
    }
  }
};

// In parallel, per critical point of args[blockIdx.y]: the strangulation
// mark of a saddle whose asc or des multiset holds one point twice (:404-417),
// and the heap entries of its des arcs, at their places in the push order.
// the entry word of critical point k: its index, dimension and boundary bit
__device__ __forceinline__ uint32_t meta_of(const SimpArgs &A, uint32_t k) {
  const uint32_t c = A.G.cellid[k];
  const int x = (int16_t)(c & 0xffff), y = (int16_t)(c >> 16);
  const bool contains = x >= A.rx0 && y >= A.ry0 && x <= A.rx1 && y <= A.ry1;
  const bool interior = x > A.rx0 && y > A.ry0 && x < A.rx1 && y < A.ry1;
  const uint32_t dim = (c & 1u) + ((c >> 16) & 1u);
  return k | (dim << 29) | (contains && !interior ? META_BOUNDARY : 0u);
}
__global__ void k_simp_meta(SimpArgs *args) {
  SimpArgs &A = args[blockIdx.y];
  const uint32_t n = A.G.ncp;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) A.meta[i] = meta_of(A, i);
}
__global__ void k_simp_prep(SimpArgs *args) {
  SimpArgs &A = args[blockIdx.y];
  const uint32_t n = A.G.ncp, base = A.doff[0];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (A.G.dim(i) == 1) {
      if ((A.aoff[i + 1] - A.aoff[i] == 2 && A.asc[A.aoff[i]] == A.asc[A.aoff[i] + 1]) ||
          (A.doff[i + 1] - A.doff[i] == 2 && A.des[A.doff[i]] == A.des[A.doff[i] + 1]))
        A.G.flags[i] |= F_STRANG;
    }
    const uint32_t mi = A.meta[i];
    for (uint32_t q = A.doff[i]; q < A.doff[i + 1]; ++q) {
      const uint32_t b = A.des[q];
      A.init[q - base] = b < n ? HeapEnt{fabsf(fsub_rn(A.fn[b], A.fn[i])), mi, A.meta[b]} : HeapEnt{0.0f, mi, b};
    }
  }
}

// A helper warp: the list edits of every cancelled pair, until told to stop.
__device__ __forceinline__ void help(const SimpArgs &a, SimpShared *sh, uint2 *stage, uint32_t runs) {
  const int who = (int)(threadIdx.x >> 5) - 1;
  WarpGraph W;
  W.G = a.G;
  W.lane = threadIdx.x & 31;
  W.stage = stage + (size_t)who * runs;
  W.nstage = runs;
  W.G.tmp_cap = a.G.tmp_cap / HELPERS;
  W.G.tmp = a.G.tmp + (size_t)who * W.G.tmp_cap;
  W.G.max_ops = ~0ull;  // (the first warp keeps the budget)
  W.team = &sh->team;
  for (;;) {
    bar_wait(BAR_GO);
    if (sh->stop) return;
    W.G.ops = 0;
    W.edit_neighbours(sh->pair, who, HELPERS);
    if (W.lane == 0) {
      if (W.G.fail) sh->team.fail = 1;
      atomicAdd(&sh->team.ops, W.G.ops);
    }
    __syncwarp();
    bar_arrive(BAR_DONE);
  }
}

// one complex per block
__global__ void __launch_bounds__(32 * SIMP_WARPS, 2) k_simplify(SimpArgs *args, int n, int levels) {
  extern __shared__ __align__(16) unsigned char heap_top[];
  __shared__ SimpShared sh;
  if (blockIdx.x >= (unsigned)n) return;
  const SimpArgs a = args[blockIdx.x];
  if (threadIdx.x == 0) {
    sh.team.top = a.G.L.top;
    sh.team.shared_top = nullptr;
    sh.team.ops = 0;
    sh.team.fail = sh.team.wrong = sh.team.late = sh.team.beat = 0;
    sh.stop = 0;
  }
  __syncthreads();
  if (threadIdx.x >= 32) {
    help(a, &sh, reinterpret_cast<uint2 *>(heap_top + ((sizeof(float) + sizeof(uint2)) << levels)), edit_runs(levels));
    return;
  }
  Simp s(a, heap_top, levels, &sh);
  s.run();
  __syncwarp();
  if (threadIdx.x == 0) {
    a.stats[3] = s.W.G.ops;
    if (s.W.G.fail) a.stats[4] |= ST_SIMPLIFY_LIMIT;
    s.W.G.L.top = sh.team.top;
    args[blockIdx.x].G = s.W.G;  // for k_unsimplify
    args[blockIdx.x].ncanc = s.ncanc;
    args[blockIdx.x].loose = s.loose;
    sh.stop = 1;
  }
  __syncwarp();
  bar_arrive(BAR_GO);
}

// un_simplify (grid_mscomplex.cpp:514-526): the cancelled pairs are
// uncancelled in reverse order, one complex per block.  A pair's
// uncancellation rewrites one asc and one des list of its own points, the asc
// list from asc lists of earlier pairs' points that no later pair changes,
// the des list from their des lists.  So the block's warps take the lists in
// order, and a warp waits only for the lists that its own one names (`ord`,
// `done`): a list is a chain of ~10 dependent memory round trips (3,200 cycles
// on one warp), and up to 16 of them overlap (2,775 pairs of a 2047x1365 field:
// 7.6 ms on one warp, 3.5 ms here).  They are taken in order, so the
// first one not yet done never waits.  A cancellation list with a pair that
// was not connected (its points may be on the list twice) goes through one
// warp in plain order.
constexpr uint32_t DONE_WORDS = 4096;  // lists tracked in shared memory, 32 a word; more: in the resubmit list's memory
__global__ void __launch_bounds__(512, 1) k_unsimplify(SimpArgs *args, int n, uint32_t stage_runs, uint32_t shared_runs) {
  extern __shared__ __align__(16) unsigned char un_smem[];
  __shared__ TeamState team;
  if (blockIdx.x >= (unsigned)n) return;
  const SimpArgs a = args[blockIdx.x];
  if (a.G.fail || a.stats[4] != 0 || a.ncanc == 0) return;  // (block-uniform)
  WarpGraph W;
  W.G = a.G;
  W.lane = threadIdx.x & 31;
  uint2 *buf = reinterpret_cast<uint2 *>(un_smem);
  W.stage = buf + (size_t)(threadIdx.x >> 5) * stage_runs;
  W.nstage = stage_runs;
  W.shared_stage = buf + (size_t)(blockDim.x >> 5) * stage_runs;
  W.nshared_stage = shared_runs;
  W.team = &team;
  const uint32_t words = (2 * a.ncanc + 31) / 32;
  W.done = words <= DONE_WORDS ? reinterpret_cast<uint32_t *>(W.shared_stage + shared_runs) : reinterpret_cast<uint32_t *>(a.resub);
  if (threadIdx.x == 0) {
    team.top = a.G.L.top;
    team.shared_top = nullptr;
    team.ops = a.G.ops;
    team.ticket = 2ull * a.ncanc;
    team.fail = team.wrong = team.late = team.beat = 0;
    team.lock = 0;
  }
  for (uint32_t i = threadIdx.x; i < a.G.ncp; i += blockDim.x) a.meta[i] = 0;
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) W.done[i] = 0;
  __syncthreads();
  if (!a.loose) {
    for (uint32_t k = threadIdx.x; k < a.ncanc; k += blockDim.x) {
      const uint2 c = a.canc[k];
      a.meta[c.x] = a.meta[c.y] = k + 1;  // (a point is cancelled once)
    }
    __syncthreads();
    W.ord = a.meta;
    W.uncancel_shared(a.canc, a.ncanc);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < a.ncanc; k += blockDim.x) {
      const uint2 c = a.canc[k];
      a.G.flags[c.x] &= ~F_CANCELLED;
      a.G.flags[c.y] &= ~F_CANCELLED;
    }
  } else if (threadIdx.x < 32) {
    for (uint32_t k = a.ncanc; k-- > 0 && !team.fail && !team.wrong;) {
      const uint2 c = a.canc[k];
      if (!W.uncancel_pairs(c.x, c.y)) team.wrong = 1;
      if (W.G.fail) team.fail = 1;
      __syncwarp();
    }
  }
  if (W.lane == 0) atomicAdd(&team.ops, W.G.ops - a.G.ops);
  __syncthreads();
  if (threadIdx.x == 0) {
    a.stats[3] = team.ops;
    if (team.late) a.stats[4] |= ST_WAIT_LIMIT;
    else if (team.wrong) a.stats[4] |= ST_INVARIANT;  // (the other warps stopped for it)
    else if (team.fail || team.ops > a.G.max_ops) a.stats[4] |= ST_SIMPLIFY_LIMIT;
  }
}

// The asc and des entries of args[blockIdx.y]'s lists.  Cancellations multiply
// counts, so a complex of a few thousand points can come to more entries than
// 32-bit offsets reach; the host refuses it before anything is sized by them.
__global__ void k_entry_sums(SimpArgs *args) {
  const SimpArgs &A = args[blockIdx.y];
  unsigned long long s[2] = {0, 0};
  const uint2 *tot = reinterpret_cast<const uint2 *>(A.G.L.total);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < A.G.ncp; i += gridDim.x * blockDim.x) {
    const uint2 t = tot[i];
    s[0] += t.x;
    s[1] += t.y;
  }
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    s[w] = warp_sum64(s[w]);
    if ((threadIdx.x & 31) == 0 && s[w]) atomicAdd(&A.stats[5 + w], s[w]);
  }
}

static cudaError_t launch_simplify(SimpArgs *args, int n, int levels, cudaStream_t st) {
  // warps and runs of scratch per block: one block per SM, or several when a batch has more complexes than SMs
  const int warps = n <= 152 ? 16 : 8;
  const uint32_t own = n <= 152 ? 1024 : 512, shared = n <= 152 ? 8192 : 4096;
  constexpr size_t un_max = sizeof(uint2) * (16 * 1024 + 8192) + sizeof(uint32_t) * DONE_WORDS;
  static SmemLimit limit, un_limit;
  cudaError_t e = limit.raise(top_bytes(TOP_LEVELS), k_simplify);
  if (e == cudaSuccess) e = un_limit.raise(un_max, k_unsimplify);
  if (e != cudaSuccess) return e;
  k_simplify<<<n, 32 * SIMP_WARPS, top_bytes(levels), st>>>(args, n, levels);
  k_unsimplify<<<n, 32 * warps, sizeof(uint2) * (warps * own + shared) + sizeof(uint32_t) * DONE_WORDS, st>>>(args, n, own, shared);
  k_entry_sums<<<dim3(n == 1 ? 64 : 4, n), 256, 0, st>>>(args);
  DMSC_LAUNCHED(3);
  return cudaGetLastError();
}

// CSR (expanded, ascending) -> run-length lists.  Capacity of a list is its
// CSR length + 4 runs; asc lists first, des lists after them.
__global__ void k_lists_from_csr(uint32_t ncp, const uint32_t *aoff, const uint32_t *asc, const uint32_t *doff,
                                 const uint32_t *des, unsigned long long des_base, uint32_t *off, uint32_t *nrun,
                                 uint32_t *cap, uint32_t *total, uint2 *pool) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ncp; i += gridDim.x * blockDim.x) {
    for (int w = 0; w < 2; ++w) {
      const uint32_t *o = w ? doff : aoff, *src = w ? des : asc;
      uint32_t b = o[i], e = o[i + 1];
      uint32_t base = w ? (uint32_t)(des_base + (unsigned long long)b + 4ull * i) : (uint32_t)(b + 4u * i);
      uint32_t m = 0;
      for (uint32_t k = b; k < e; ++k) {
        if (m > 0 && pool[base + m - 1].x == src[k]) pool[base + m - 1].y += 1;
        else pool[base + m++] = make_uint2(src[k], 1u);
      }
      off[2 * i + w] = base; nrun[2 * i + w] = m; cap[2 * i + w] = (e - b) + 4; total[2 * i + w] = e - b;
    }
  }
}

// run-length lists -> expanded CSR (offsets from a scan of the totals; a list
// never writes past the next list's offset).  Counts multiply over a long
// simplification (42 million entries in lists of 4,000 points on one 256x256
// field), so the work goes by the entries: a short list is written by its
// thread, a longer one by its warp, 32 runs at a time, and of those a run of
// more than FILL_RUN entries in pieces that k_fill writes, a block each (the
// 42 million entries: 299 ms with a thread per list, 0.5 ms here).
constexpr uint32_t FILL_RUN = 1024, FILL_PIECE = 16384;
struct FillPiece {
  uint32_t value, at, n;
};
static size_t fill_room(unsigned long long entries) { return entries / FILL_RUN + 16; }  // pieces: each, or the run it ends, is longer
__global__ void __launch_bounds__(256) k_csr_from_lists(uint32_t ncp, const uint32_t *off, const uint32_t *nrun, const uint2 *pool, int which,
                                                        const uint32_t *outoff, uint32_t *out, FillPiece *pieces, uint32_t *npieces, uint32_t room) {
  const int lane = threadIdx.x & 31;
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < ncp; i0 += step) {
    const uint32_t i = i0 + lane;
    uint32_t o = 0, end = 0, n = 0, src = 0;
    if (i < ncp) {
      o = outoff[i];
      end = outoff[i + 1];
      n = nrun[2 * i + which];
      src = off[2 * i + which];
    }
    const bool small = end - o <= 16;
    if (small)
      for (uint32_t k = 0; k < n; ++k) {
        const uint2 r = pool[src + k];
        for (uint32_t c = 0; c < r.y && o < end; ++c) out[o++] = r.x;
      }
    for (unsigned big = __ballot_sync(FULL_WARP, !small); big; big &= big - 1) {
      const int s = __ffs(big) - 1;
      uint32_t at = __shfl_sync(FULL_WARP, o, s);
      const uint32_t e = __shfl_sync(FULL_WARP, end, s), m = __shfl_sync(FULL_WARP, n, s), p = __shfl_sync(FULL_WARP, src, s);
      for (uint32_t k0 = 0; k0 < m && at < e; k0 += 32) {
        uint2 r = make_uint2(0, 0);
        if (k0 + lane < m) r = pool[p + k0 + lane];
        uint32_t all;  // (a list's counts add up to its length)
        const uint32_t x = at + warp_exscan(r.y, lane, all);
        const uint32_t cnt = x >= e || x < at ? 0u : min(r.y, e - x);
        if (cnt > FILL_RUN) {  // whole pieces of the run
          const uint32_t q = (cnt + FILL_PIECE - 1) / FILL_PIECE, w = atomicAdd(npieces, q);
          for (uint32_t c = 0; c < q && w + c < room; ++c)
            pieces[w + c] = FillPiece{r.x, x + c * FILL_PIECE, min(FILL_PIECE, cnt - c * FILL_PIECE)};
        } else if (cnt <= 4) {
          for (uint32_t c = 0; c < cnt; ++c) out[x + c] = r.x;
        }
        for (unsigned mid = __ballot_sync(FULL_WARP, cnt > 4 && cnt <= FILL_RUN); mid; mid &= mid - 1) {
          const int u = __ffs(mid) - 1;
          const uint32_t v = __shfl_sync(FULL_WARP, r.x, u), to = __shfl_sync(FULL_WARP, x, u), c1 = __shfl_sync(FULL_WARP, cnt, u);
          for (uint32_t c = lane; c < c1; c += 32) out[to + c] = v;
        }
        at += all;
      }
    }
  }
}
__global__ void __launch_bounds__(256) k_fill(const FillPiece *pieces, const uint32_t *npieces, uint32_t room, uint32_t *out) {
  const uint32_t n = min(*npieces, room);
  for (uint32_t b = blockIdx.x; b < n; b += gridDim.x) {
    const FillPiece p = pieces[b];
    for (uint32_t c = threadIdx.x; c < p.n; c += blockDim.x) out[p.at + c] = p.value;
  }
}
__global__ void k_pick_len(uint32_t ncp, const uint32_t *len, int which, uint32_t *out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ncp; i += gridDim.x * blockDim.x) out[i] = len[2 * i + which];
}

static unsigned blocks_for(long long n) {
  long long b = (n + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  return (unsigned)(b < 1 ? 1 : b);
}

// Work buffers of one simplification (one stream-ordered allocation).
struct SimplifyWork {
  SimpArgs a;
  char *buf = nullptr;
  uint8_t *flags_in = nullptr;     // caller's arrays, written back on success
  uint32_t *pair_in = nullptr;
  uint32_t *lens = nullptr;        // ncp words for the rebuilt offsets
};

cudaError_t simplify_run(SimplifyIO &io, cudaStream_t st) {
  const uint32_t ncp = (uint32_t)io.ncp;
  unsigned long long des_base = (unsigned long long)io.nasc + 4ull * ncp;
  unsigned long long base_top = des_base + (unsigned long long)io.ndes + 4ull * ncp;
  const unsigned long long pool_cap = base_top + 2 * base_top + (1ull << 22);
  const unsigned long long heap_cap = std::min(4ull * io.ndes + (1ull << 20), HEAP_MAX);
  // scratch runs: two per added value of a merged list (edit_list), per helper warp
  const unsigned long long tmp_cap = std::max(1ull << 22, 2ull * HELPERS * ncp);
  if (pool_cap > 0xffffffffull) return cudaErrorInvalidValue;  // list offsets are 32-bit
  if (ncp > IDX_MASK) return cudaErrorInvalidValue;               // heap entries hold 29-bit indices
  auto rnd = [](size_t n) { return (n + 255) / 256 * 256; };
  size_t sizes[] = {sizeof(uint32_t) * 2 * ncp, sizeof(uint32_t) * 2 * ncp, sizeof(uint32_t) * 2 * ncp,
                    sizeof(uint32_t) * 2 * ncp, sizeof(uint2) * pool_cap, sizeof(uint2) * tmp_cap, sizeof(float) * (heap_cap + 2),
                    sizeof(uint2) * (heap_cap + 2), sizeof(HeapEnt) * heap_cap, sizeof(uint2) * (ncp + 1), sizeof(unsigned long long) * 8,
                    sizeof(uint8_t) * (ncp + 1), sizeof(uint32_t) * (ncp + 1), sizeof(uint32_t) * (ncp + 1),
                    sizeof(HeapEnt) * ((size_t)io.ndes + 1), sizeof(SimpArgs), sizeof(uint32_t) * (ncp + 1)};
  size_t bytes = 0;
  for (size_t z : sizes) bytes += rnd(z);
  SimplifyWork *w = new SimplifyWork;
  io.work = w;
  cudaError_t e = cudaMallocAsync((void **)&w->buf, bytes, st);
  if (e != cudaSuccess) { w->buf = nullptr; return e; }
  char *p = w->buf;
  int si = 0;
  auto take = [&]() { char *r = p; p += rnd(sizes[si++]); return r; };
  SimpArgs &a = w->a;
  Graph &G = a.G;
  G.ncp = ncp;
  G.cellid = const_cast<uint32_t *>(io.cellid);
  a.fn = io.fn;
  G.L.off = (uint32_t *)take();
  G.L.nrun = (uint32_t *)take();
  G.L.cap = (uint32_t *)take();
  G.L.total = (uint32_t *)take();
  G.L.pool = (uint2 *)take();
  G.L.top = base_top;
  G.L.pool_cap = pool_cap;
  G.tmp = (uint2 *)take();
  G.tmp_cap = tmp_cap;
  a.hkey = (float *)take();
  a.hab = (uint2 *)take();
  a.heap_cap = heap_cap;
  a.resub = (HeapEnt *)take();
  a.canc = (uint2 *)take();
  a.stats = (unsigned long long *)take();
  G.flags = (uint8_t *)take();
  G.pair_idx = (uint32_t *)take();
  w->lens = (uint32_t *)take();
  a.init = (HeapEnt *)take();
  a.ninit = (unsigned long long)io.ndes;
  a.aoff = io.aoff; a.asc = io.asc; a.doff = io.doff; a.des = io.des;
  SimpArgs *dargs = (SimpArgs *)take();
  a.meta = (uint32_t *)take();
  w->flags_in = io.flags;
  w->pair_in = io.pair_idx;
  a.rx0 = io.rect[0]; a.ry0 = io.rect[1]; a.rx1 = io.rect[2]; a.ry1 = io.rect[3];
  a.tresh = io.tresh;
  G.max_ops = io.max_ops;
  G.ops = 0;
  G.fail = false;
  e = cudaMemsetAsync(a.stats, 0, sizeof(unsigned long long) * 8, st);
  if (e == cudaSuccess && ncp) e = cudaMemcpyAsync(G.flags, io.flags, ncp, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess && ncp) e = cudaMemcpyAsync(G.pair_idx, io.pair_idx, 4ull * ncp, cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) return e;
  if (ncp) {
    k_lists_from_csr<<<blocks_for(ncp), 256, 0, st>>>(ncp, io.aoff, io.asc, io.doff, io.des, des_base, G.L.off,
                                                       G.L.nrun, G.L.cap, G.L.total, G.L.pool);
    DMSC_LAUNCHED(1);
    e = cudaMemcpyAsync(dargs, &a, sizeof(SimpArgs), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    k_simp_meta<<<blocks_for(ncp), 256, 0, st>>>(dargs);
    k_simp_prep<<<blocks_for(ncp), 256, 0, st>>>(dargs);
    DMSC_LAUNCHED(2);
    if ((e = launch_simplify(dargs, 1, TOP_LEVELS, st)) != cudaSuccess) return e;
  }
  e = cudaMemcpyAsync(io.host_stats, a.stats, sizeof(unsigned long long) * 7, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && io.host_stats[4] == 0 && std::max(io.host_stats[5], io.host_stats[6]) > 0xffffffffull)
    io.host_stats[4] = ST_TOO_LONG;
  if (e != cudaSuccess || io.host_stats[4] != 0 || !ncp) return e;
  // new CSR offsets (asc, then des) from the list lengths
  for (int which = 0; which < 2 && e == cudaSuccess; ++which) {
    uint32_t *offs = which ? io.doff : io.aoff;
    k_pick_len<<<blocks_for(ncp), 256, 0, st>>>(ncp, G.L.total, which, w->lens);
    DMSC_LAUNCHED(1);
    e = scan_exclusive_u32(w->lens, ncp, offs, offs + ncp, st);
  }
  uint32_t tot[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[0], io.aoff + ncp, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[1], io.doff + ncp, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  io.nasc_out = tot[0];
  io.ndes_out = tot[1];
  return e;
}

// The lists of kind `which` (0 asc, 1 des) into out; entries: at most that many.
static cudaError_t emit_lists(uint32_t ncp, const uint32_t *off, const uint32_t *nrun, const uint2 *pool, int which,
                              const uint32_t *outoff, uint32_t *out, unsigned long long entries, cudaStream_t st) {
  const size_t room = entries > FILL_RUN ? fill_room(entries) : 0;  // (no run can be long enough)
  char *buf = nullptr;
  cudaError_t e = cudaSuccess;
  if (room) {
    if ((e = cudaMallocAsync((void **)&buf, 16 + sizeof(FillPiece) * room, st)) != cudaSuccess) return e;
    e = cudaMemsetAsync(buf, 0, 4, st);
  }
  uint32_t *n = (uint32_t *)buf;
  FillPiece *pieces = (FillPiece *)(buf + 16);
  k_csr_from_lists<<<blocks_for(ncp), 256, 0, st>>>(ncp, off, nrun, pool, which, outoff, out, pieces, n, (uint32_t)room);
  DMSC_LAUNCHED(1);
  if (room) {
    k_fill<<<(unsigned)std::min<size_t>(room, 152 * 8), 256, 0, st>>>(pieces, n, (uint32_t)room, out);
    DMSC_LAUNCHED(1);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (buf) cudaFreeAsync(buf, st);
  return e;
}

cudaError_t simplify_emit(SimplifyIO &io, uint32_t *asc, uint32_t *des, cudaStream_t st) {
  SimplifyWork *w = (SimplifyWork *)io.work;
  const uint32_t ncp = (uint32_t)io.ncp;
  if (!w || !ncp) return cudaSuccess;
  const Lists &L = w->a.G.L;
  cudaError_t e = emit_lists(ncp, L.off, L.nrun, L.pool, 0, io.aoff, asc, (unsigned long long)io.nasc_out, st);
  if (e == cudaSuccess) e = emit_lists(ncp, L.off, L.nrun, L.pool, 1, io.doff, des, (unsigned long long)io.ndes_out, st);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(w->flags_in, w->a.G.flags, ncp, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->pair_in, w->a.G.pair_idx, 4ull * ncp, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e;
}

void simplify_release(SimplifyIO &io, cudaStream_t st) {
  SimplifyWork *w = (SimplifyWork *)io.work;
  if (!w) return;
  if (w->buf) cudaFreeAsync(w->buf, st);
  delete w;
  io.work = nullptr;
}

// ---------------------------------------------------------------------------
// batches: one block per complex to simplify, all in one launch
// ---------------------------------------------------------------------------
struct BatchSimplifyWork {
  char *buf = nullptr;
  uint32_t *off = nullptr, *nrun = nullptr, *lcap = nullptr, *total = nullptr, *lens = nullptr;
  uint2 *pool = nullptr;
  SimpArgs *dargs = nullptr;
  unsigned long long *dstats = nullptr;
  int nsimp = 0;
};

cudaError_t simplify_batch_run(BatchSimplifyIO &io, cudaStream_t st) {
  const uint32_t ncp = (uint32_t)io.ncp;
  const unsigned long long des_base = (unsigned long long)io.nasc + 4ull * ncp;
  const unsigned long long base_top = des_base + (unsigned long long)io.ndes + 4ull * ncp;
  // per simplified grid: pool growth region, heap, resubmits, cancellations, scratch runs
  std::vector<int> which;
  unsigned long long grow = 0, heap = 0, canc = 0, tmp = 0, init = 0;
  const unsigned long long sc = io.scale ? io.scale : 1;
  auto grow_of = [&](unsigned long long na, unsigned long long nd, unsigned long long n) {
    return sc * (4 * (na + nd + 8 * n) + 16384);
  };
  auto heap_of = [&](unsigned long long nd) { return std::min(sc * (8 * nd + 16384), HEAP_MAX); };  // (even)
  auto tmp_of = [&](unsigned long long na, unsigned long long nd, unsigned long long n) {
    return sc * (4 * (na + nd) + 16384) + 2 * HELPERS * n;
  };
  for (int g = 0; g < io.ngrids; ++g) {
    const unsigned long long n = io.cpb[g + 1] - io.cpb[g];
    if (!(io.tresh[g] > 0.0) || n == 0) continue;
    const unsigned long long na = io.abase[g + 1] - io.abase[g], nd = io.dbase[g + 1] - io.dbase[g];
    which.push_back(g);
    grow += grow_of(na, nd, n);
    heap += heap_of(nd) + 2;
    canc += n + 1;
    tmp += tmp_of(na, nd, n);
    init += nd + 1;
  }
  const unsigned long long pool_cap = base_top + grow;
  if (pool_cap > 0xffffffffull) return cudaErrorInvalidValue;  // list offsets are 32-bit
  // Blocks start roughly in index order and more grids than fit at once wait
  // for a free slot, while the batch lasts as long as its longest replay: the
  // complexes with the most arcs (the longest replays, as a rule) take the
  // first blocks.
  std::stable_sort(which.begin(), which.end(), [&](int x, int y) {
    const unsigned long long ax = (io.abase[x + 1] - io.abase[x]) + (io.dbase[x + 1] - io.dbase[x]);
    const unsigned long long ay = (io.abase[y + 1] - io.abase[y]) + (io.dbase[y + 1] - io.dbase[y]);
    return ax > ay;
  });
  const int ns = (int)which.size();
  auto rnd = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t sizes[] = {4ull * 2 * ncp, 4ull * 2 * ncp, 4ull * 2 * ncp, 4ull * 2 * ncp, 4ull * (ncp + 1),
                          sizeof(uint2) * pool_cap, sizeof(uint2) * tmp, sizeof(float) * heap, sizeof(uint2) * heap,
                          sizeof(HeapEnt) * heap,
                          sizeof(uint2) * canc, sizeof(unsigned long long) * 8 * (size_t)(ns + 1),
                          sizeof(SimpArgs) * (size_t)(ns + 1), sizeof(HeapEnt) * (init + 1), 4ull * (ncp + 1)};
  size_t bytes = 0;
  for (size_t z : sizes) bytes += rnd(z);
  BatchSimplifyWork *w = new BatchSimplifyWork;
  io.work = w;
  cudaError_t e = cudaMallocAsync((void **)&w->buf, bytes, st);
  if (e != cudaSuccess) { w->buf = nullptr; return e; }
  char *p = w->buf;
  int si = 0;
  auto take = [&]() { char *r = p; p += rnd(sizes[si++]); return r; };
  w->off = (uint32_t *)take(); w->nrun = (uint32_t *)take(); w->lcap = (uint32_t *)take(); w->total = (uint32_t *)take();
  w->lens = (uint32_t *)take();
  w->pool = (uint2 *)take();
  uint2 *dtmp = (uint2 *)take();
  float *dhkey = (float *)take();
  uint2 *dhab = (uint2 *)take();
  HeapEnt *dres = (HeapEnt *)take();
  uint2 *dcanc = (uint2 *)take();
  w->dstats = (unsigned long long *)take();
  w->dargs = (SimpArgs *)take();
  HeapEnt *dinit = (HeapEnt *)take();
  uint32_t *dmeta = (uint32_t *)take();
  w->nsimp = ns;
  if (ncp) {
    k_lists_from_csr<<<blocks_for(ncp), 256, 0, st>>>(ncp, io.aoff, io.asc, io.doff, io.des, des_base, w->off, w->nrun,
                                                       w->lcap, w->total, w->pool);
    DMSC_LAUNCHED(1);
  }
  e = cudaMemsetAsync(w->dstats, 0, sizeof(unsigned long long) * 8 * (size_t)(ns + 1), st);
  std::vector<SimpArgs> args(ns);
  unsigned long long top = base_top, ho = 0, co = 0, to = 0, io2 = 0;
  for (int k = 0; k < ns && e == cudaSuccess; ++k) {
    const int g = which[k];
    const unsigned long long c0 = io.cpb[g], n = io.cpb[g + 1] - c0;
    const unsigned long long na = io.abase[g + 1] - io.abase[g], nd = io.dbase[g + 1] - io.dbase[g];
    SimpArgs &a = args[k];
    Graph &G = a.G;
    G = Graph();
    G.ncp = (uint32_t)n;
    G.cellid = const_cast<uint32_t *>(io.cellid) + c0;
    G.flags = io.flags + c0;
    G.pair_idx = io.pair_idx + c0;
    G.L.off = w->off + 2 * c0; G.L.nrun = w->nrun + 2 * c0; G.L.cap = w->lcap + 2 * c0; G.L.total = w->total + 2 * c0;
    G.L.pool = w->pool;
    G.L.top = top;
    top += grow_of(na, nd, n);
    G.L.pool_cap = top;
    G.tmp = dtmp + to;
    G.tmp_cap = tmp_of(na, nd, n);
    to += G.tmp_cap;
    G.max_ops = io.max_ops;
    G.ops = 0;
    G.fail = false;
    a.fn = io.fn + c0;
    a.meta = dmeta + c0;
    a.hkey = dhkey + ho;
    a.hab = dhab + ho;
    a.resub = dres + ho;
    a.heap_cap = heap_of(nd);
    ho += a.heap_cap + 2;
    a.canc = dcanc + co;
    co += n + 1;
    a.aoff = io.aoff + c0; a.asc = io.asc; a.doff = io.doff + c0; a.des = io.des;
    a.init = dinit + io2;
    a.ninit = nd;
    io2 += nd + 1;
    a.rx0 = io.rect[4 * g]; a.ry0 = io.rect[4 * g + 1]; a.rx1 = io.rect[4 * g + 2]; a.ry1 = io.rect[4 * g + 3];
    a.tresh = io.tresh[g];
    a.stats = w->dstats + 8 * k;
  }
  if (e == cudaSuccess && ns) e = cudaMemcpyAsync(w->dargs, args.data(), sizeof(SimpArgs) * ns, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && ns) {
    // one grid per SM can keep 14 heap levels in shared memory; more grids
    // than SMs keep 13, two per SM (a batch of 1000 grids, two sets of inputs:
    // 13 levels 46.0 and 53.1 ms, 12 levels (three per SM) 48.3 and 57.2, 14
    // levels 55.1 and 44.1: it depends on which replay is the longest)
    const int levels = ns <= 152 ? TOP_LEVELS : TOP_LEVELS_BATCH;
    k_simp_meta<<<dim3(64, (unsigned)ns), 256, 0, st>>>(w->dargs);
    k_simp_prep<<<dim3(64, (unsigned)ns), 256, 0, st>>>(w->dargs);
    DMSC_LAUNCHED(2);
    e = launch_simplify(w->dargs, ns, levels, st);
  }
  std::vector<unsigned long long> hs(8 * (size_t)(ns + 1), 0);
  if (e == cudaSuccess && ns) e = cudaMemcpyAsync(hs.data(), w->dstats, sizeof(unsigned long long) * 8 * ns, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  for (int g = 0; g < io.ngrids; ++g)
    for (int q = 0; q < 5; ++q) io.host_stats[5 * g + q] = 0;
  for (int k = 0; k < ns; ++k)
    for (int q = 0; q < 5; ++q) io.host_stats[5 * which[k] + q] = hs[8 * k + q];
  // a grid whose lists outgrow 32-bit offsets fails alone; so does every
  // further one once the batch's lists together would
  unsigned long long tot[2] = {(unsigned long long)io.nasc, (unsigned long long)io.ndes};
  for (int k = 0; k < ns; ++k) {
    const int g = which[k];
    const unsigned long long na = hs[8 * k + 5], nd = hs[8 * k + 6];
    const unsigned long long a0 = io.abase[g + 1] - io.abase[g], d0 = io.dbase[g + 1] - io.dbase[g];
    if (hs[8 * k + 4] != 0) continue;
    if (tot[0] - a0 + na > 0xffffffffull || tot[1] - d0 + nd > 0xffffffffull) {
      io.host_stats[5 * g + 4] = ST_TOO_LONG;
      continue;
    }
    tot[0] += na - a0;
    tot[1] += nd - d0;
  }
  return cudaSuccess;  // the caller reads the per-grid status
}

// List offsets of the simplified batch; the grids in `dead` (whose
// simplification failed) keep their critical points but get empty lists.
cudaError_t simplify_batch_offsets(BatchSimplifyIO &io, const std::vector<int> &dead, cudaStream_t st) {
  BatchSimplifyWork *w = (BatchSimplifyWork *)io.work;
  const uint32_t ncp = (uint32_t)io.ncp;
  io.nasc_out = io.ndes_out = 0;
  if (!w || !ncp) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  for (int g : dead) {  // no runs and no total: the emit writes nothing for them
    const unsigned long long c0 = io.cpb[g], n = io.cpb[g + 1] - c0;
    if (n && e == cudaSuccess) e = cudaMemsetAsync(w->total + 2 * c0, 0, 8ull * n, st);
    if (n && e == cudaSuccess) e = cudaMemsetAsync(w->nrun + 2 * c0, 0, 8ull * n, st);
  }
  for (int wch = 0; wch < 2 && e == cudaSuccess; ++wch) {
    uint32_t *offs = wch ? io.doff : io.aoff;
    k_pick_len<<<blocks_for(ncp), 256, 0, st>>>(ncp, w->total, wch, w->lens);
    DMSC_LAUNCHED(1);
    e = scan_exclusive_u32(w->lens, ncp, offs, offs + ncp, st);
  }
  uint32_t tot[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[0], io.aoff + ncp, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&tot[1], io.doff + ncp, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  io.nasc_out = tot[0];
  io.ndes_out = tot[1];
  return e;
}

cudaError_t simplify_batch_emit(BatchSimplifyIO &io, uint32_t *asc, uint32_t *des, cudaStream_t st) {
  BatchSimplifyWork *w = (BatchSimplifyWork *)io.work;
  const uint32_t ncp = (uint32_t)io.ncp;
  if (!w || !ncp) return cudaSuccess;
  cudaError_t e = emit_lists(ncp, w->off, w->nrun, w->pool, 0, io.aoff, asc, (unsigned long long)io.nasc_out, st);
  if (e == cudaSuccess) e = emit_lists(ncp, w->off, w->nrun, w->pool, 1, io.doff, des, (unsigned long long)io.ndes_out, st);
  return e;
}

void simplify_batch_release(BatchSimplifyIO &io, cudaStream_t st) {
  BatchSimplifyWork *w = (BatchSimplifyWork *)io.work;
  if (!w) return;
  if (w->buf) cudaFreeAsync(w->buf, st);
  delete w;
  io.work = nullptr;
}

}  // namespace dmsc
