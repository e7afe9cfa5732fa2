// warp_graph.cuh -- cancel_pairs and uncancel_pairs of msc_graph.cuh by warps.
//
// The order-dependent passes (the simplification's replay, the merges'
// boundary steps) change the graph one pair at a time, and each change is a
// handful of list edits whose cost is dependent memory round trips.  A pair's
// edits all concern different lists (the neighbours' asc lists and des lists,
// and a cell's lists hold cells of one dimension), so they are made side by
// side: up to 32 short lists (at most 8 runs, at most one added value) by one
// warp, a list per lane, each read once into registers, edited there and
// written back; a longer list by all lanes of a warp together, one merge for
// all added values and the removed one.  Every list is left with the runs the
// one-thread functions leave, and the operation count (`ops`) grows by the
// same amount.
//
// A cancellation is orient (which point's asc list holds the other), then
// edit_neighbours by all warps of a team, and close; an uncancellation is
// uncancel_list for each of its two lists, by one warp (uncancel_pairs) or as
// tasks that a team's warps take (uncancel_shared).
//
// All lanes call every member function together with the same arguments and
// hold the same copy of the graph's descriptor.
#pragma once
#include "msc_graph.cuh"

namespace dmsc {

constexpr unsigned FULL_WARP = 0xffffffffu;

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
  if (!__any_sync(FULL_WARP, v >= (1ull << 27))) return __reduce_add_sync(FULL_WARP, (uint32_t)v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_WARP, v, o);
  return v;
}
__device__ __forceinline__ uint32_t warp_exscan(uint32_t v, int lane, uint32_t &total) {
  uint32_t s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL_WARP, s, o);
    if (lane >= o) s += t;
  }
  total = __shfl_sync(FULL_WARP, s, 31);
  return s - v;
}

// What the warps of a block that edit one graph side by side share.
struct TeamState {
  unsigned long long top;    // the list pool's top
  unsigned long long ops;    // operations the warps have reported
  unsigned long long ticket; // pairs not yet taken
  uint32_t fail, wrong;      // a pool, budget or wait ran out; a reference logic_error condition
  int lock;                  // 1: a warp uses the scratch all warps share
  uint32_t late;             // a wait on another warp ran out (fail is set too)
  uint32_t beat;             // parts done of lists that take long
  unsigned long long *shared_top;  // the pool's top where several blocks edit the graph (then top is unused)
};
// A wait on another warp polls so often, then looks whether the team got on
// since the last time it looked: whether a task was taken, or the beat moved.
// If neither, it gives up.  (A list may take longer than the polls to rewrite:
// millions of values are sorted by one warp in global memory, at worst by one
// lane.  Its loops count a beat at least every few ms; lists of usual lengths
// have none.)  The look is outside the loop of the polls: within it, it took 5%
// of the time of all uncancellations.
#ifndef DMSC_WAIT_POLLS
#define DMSC_WAIT_POLLS (1ull << 26)
#endif
constexpr unsigned long long WAIT_LIMIT = DMSC_WAIT_POLLS;
constexpr uint32_t BEAT_STEPS = 4096;  // a loop over a list counts a beat after so many steps (a power of two)
constexpr int BAR_EDIT = 3;

struct WarpGraph {
  Graph G;        // the same in every lane
  int lane;
  uint2 *stage;   // scratch in shared memory for `nstage` runs (a power of two; may be null)
  uint32_t nstage;
  // several warps on one graph: the shared state; side-by-side uncancellation:
  // the points' pairs, the lists done, and scratch in shared memory that one
  // warp at a time takes
  TeamState *team = nullptr;
  const uint32_t *ord = nullptr;  // 1 + place of the point's pair on the cancellation list, 0 for points of no pair
  uint32_t *done = nullptr;       // a bit per rewritten list: 2 * place of the pair + (0 asc, 1 des)
  uint2 *shared_stage = nullptr;
  uint32_t nshared_stage = 0;

  __device__ __forceinline__ unsigned lt() const { return (1u << lane) - 1u; }
  // by the calling lane: its warp has done a part of a long list
  __device__ __forceinline__ void moved_on() const {
    if (team) atomicAdd(&team->beat, 1u);
  }
  // another warp's work has failed
  __device__ __forceinline__ bool called_off() const {
    return *(volatile uint32_t *)&team->fail || *(volatile uint32_t *)&team->wrong;
  }
  // All lanes, after a wait that was called off or whose polls ran out: whether
  // to wait on, as the team got on since the last time (seen: what it had done
  // then, ~0 the first time).
  __device__ __forceinline__ bool wait_on(unsigned long long &seen) const {
    uint32_t now = *(volatile uint32_t *)&team->beat - (uint32_t)*(volatile unsigned long long *)&team->ticket;  // (tasks count down)
    now = __shfl_sync(FULL_WARP, now, 0);
    if (__any_sync(FULL_WARP, called_off())) return false;
    if (seen == now) {
      if (lane == 0) *(volatile uint32_t *)&team->late = 1;
      return false;
    }
    seen = now;
    return true;
  }

  // first run of p[0..n) (ascending values) with value >= x
  __device__ __forceinline__ uint32_t lower(const uint2 *p, uint32_t n, uint32_t x) const {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 32) {  // 32 probes a round
      const uint32_t step = (hi - lo) / 33;
      const unsigned b = __ballot_sync(FULL_WARP, p[lo + step * (lane + 1)].x < x);
      const uint32_t c = __popc(b);
      if (c < 32) hi = lo + step * (c + 1);
      if (c) lo = lo + step * c + 1;
    }
    const unsigned b = __ballot_sync(FULL_WARP, (uint32_t)lane < hi - lo && p[lo + lane].x < x);
    return lo + __popc(b);
  }
  __device__ __forceinline__ bool holds(const uint2 *p, uint32_t n, uint32_t x) const {
    if (n <= 32) return __any_sync(FULL_WARP, (uint32_t)lane < n && p[lane].x == x);
    const uint32_t i = lower(p, n, x);
    return i < n && p[i].x == x;
  }
  __device__ __forceinline__ void mark(uint32_t a, uint32_t d) const {
    G.flags[a] |= F_STRANG;
    G.flags[d] |= F_STRANG;
  }

  // List l loses r's run (has_r) and takes, with counts mult * y, the runs of
  // S[0..sn) but `skip`'s.  mark_a: a value whose count reaches 2 is marked
  // strangulated together with list l's point.  Counts the shifts the single
  // inserts and the erase would make, and with mark_a the counts taken.
  __device__ __forceinline__ void edit_list(uint32_t l, uint32_t n, uint32_t cap, uint32_t tot, uint32_t off0,
                                            const uint2 *S, uint32_t sn, uint32_t skip, uint32_t mult, bool has_r,
                                            uint32_t r, bool mark_a) {
    uint2 *p = G.L.pool + off0;
    if (n <= 32 && sn <= 32) {  // a run and an added value per lane, in registers
      uint2 v = make_uint2(0xffffffffu, 0u), s = make_uint2(skip, 0u);
      if ((uint32_t)lane < n) v = p[lane];
      if ((uint32_t)lane < sn) s = S[lane];
      const bool valid = s.x != skip;
      const unsigned long long c = (unsigned long long)s.y * mult;
      if (!__any_sync(FULL_WARP, valid && c >= (1u << 24))) {
        // runs below this lane's value, and whether the value has a run
        uint32_t pos = 0;
        bool dup = false;
#pragma unroll 4
        for (uint32_t i = 0; i < n; ++i) {
          if (sn == 0) break;
          const uint32_t xi = __shfl_sync(FULL_WARP, v.x, i);
          pos += xi < s.x;
          dup |= xi == s.x;
        }
        const bool fresh = valid && !dup;
        dup = valid && dup;
        // added runs below this lane's run
        const uint32_t sx = fresh ? s.x : 0xffffffffu;
        uint32_t sh = 0;
#pragma unroll 4
        for (uint32_t j = 0; j < sn; ++j) sh += __shfl_sync(FULL_WARP, sx, j) < v.x;
        bool bad = false;
        if (__any_sync(FULL_WARP, dup))
          for (uint32_t j = 0; j < sn; ++j) {
            const uint32_t xj = __shfl_sync(FULL_WARP, dup ? s.x : 0xffffffffu, j), cj = __shfl_sync(FULL_WARP, (uint32_t)c, j);
            if (v.x == xj && (uint32_t)lane < n) {
              if (v.y > 0xffffffffu - cj) bad = true;
              v.y += cj;
            }
          }
        const unsigned fm = __ballot_sync(FULL_WARP, fresh);
        const uint32_t knew = __popc(fm);
        const bool ex = has_r && __any_sync(FULL_WARP, v.x == r);
        const uint32_t m = n + knew - (ex ? 1u : 0u);
        const uint32_t add = __reduce_add_sync(FULL_WARP, valid ? (uint32_t)c : 0u);
        unsigned long long ticks = __reduce_add_sync(FULL_WARP, fresh ? n - pos : 0u);
        uint32_t ey = 0;
        if (ex) {
          ey = __reduce_max_sync(FULL_WARP, v.x == r ? v.y : 0u);
          ticks += n + knew - __reduce_add_sync(FULL_WARP, (v.x < r ? 1u : 0u) + (sx < r ? 1u : 0u));
        }
        if (mark_a) {
          ticks += add;
          if (dup || (valid && c >= 2)) mark(l >> 1, s.x);
        }
        if (__any_sync(FULL_WARP, bad) || tot > 0xffffffffu - add) { G.fail = true; return; }
        uint32_t off = off0;
        if (m > cap && !grow(l, cap, m, off)) return;
        p = G.L.pool + off;
        if ((uint32_t)lane < n && !(ex && v.x == r)) p[lane + sh - (ex && v.x > r ? 1u : 0u)] = v;
        if (fresh) p[pos + __popc(fm & lt()) - (ex && s.x > r ? 1u : 0u)] = make_uint2(s.x, (uint32_t)c);
        if (lane == 0) { G.L.nrun[l] = m; G.L.total[l] = tot + add - ey; }
        __syncwarp();
        G.tick(ticks);
        return;
      }
    }
    // up to four values: eight runs a lane, all in flight at once, and each value's
    // place from ballots (a list of 100 runs: 3300 cycles by the searches and
    // moves below, 1000 so)
    if (n <= 256 && sn <= 4) {
      constexpr int K = 8;
      uint2 v[K], s = make_uint2(skip, 0u);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        v[k] = make_uint2(0xffffffffu, 0u);
        if (k * 32u + lane < n) v[k] = p[k * 32 + lane];
      }
      if ((uint32_t)lane < sn) s = S[lane];
      uint32_t e = n, ey = 0;
      if (has_r) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (k * 32u >= n) break;
          const unsigned b = __ballot_sync(FULL_WARP, v[k].x == r);
          if (b) {
            e = k * 32 + __ffs(b) - 1;
            ey = __shfl_sync(FULL_WARP, v[k].y, __ffs(b) - 1);
          }
        }
      }
      const bool ex = e < n;
      uint32_t at[4], fresh = 0, changed = 0, ebef = 0, pos = 0;  // places of the added runs (n: none there)
      unsigned long long ticks = 0, add = 0;
      bool bad = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        at[j] = 0xffffffffu;
        if (j >= (int)sn) continue;
        const uint32_t x = __shfl_sync(FULL_WARP, s.x, j);
        if (x == skip) continue;
        const unsigned long long c = (unsigned long long)__shfl_sync(FULL_WARP, s.y, j) * mult;
        if (c > 0xffffffffull) bad = true;
        uint32_t below = 0;
        bool here = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (k * 32u >= n) break;
          below += __popc(__ballot_sync(FULL_WARP, v[k].x < x));
          if (v[k].x == x) {
            here = true;
            if (v[k].y > 0xffffffffu - (uint32_t)c) bad = true;
            v[k].y += (uint32_t)c;
            changed |= 1u << k;
          }
        }
        const bool dup = __any_sync(FULL_WARP, here);
        if (!dup) {
          at[j] = below;
          fresh |= 1u << j;
          ticks += n - below;
          ebef += x < r ? 1u : 0u;
          if (lane == j) pos = below;
        }
        add += c;
        if (mark_a && lane == j && (dup || c >= 2)) mark(l >> 1, x);
      }
      if (mark_a) ticks += add;
      const uint32_t knew = __popc(fresh), m = n + knew - (ex ? 1u : 0u);
      if (ex) ticks += n + knew - (e + ebef);
      if (__any_sync(FULL_WARP, bad) || tot + add > 0xffffffffull) { G.fail = true; return; }
      uint32_t off = off0;
      if (m > cap && !grow(l, cap, m, off)) return;
      uint2 *const dst = G.L.pool + off;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k * 32u >= n) break;
        const uint32_t i = k * 32 + lane;
        const uint32_t to = i + (at[0] <= i) + (at[1] <= i) + (at[2] <= i) + (at[3] <= i) - (ex && i > e ? 1u : 0u);
        if (i < n && i != e && (dst != p || to != i || (changed >> k & 1))) dst[to] = v[k];
      }
      if (fresh >> lane & 1)
        dst[pos + __popc(fresh & lt()) - (ex && e < pos ? 1u : 0u)] = make_uint2(s.x, (uint32_t)((unsigned long long)s.y * mult));
      if (lane == 0) { G.L.nrun[l] = m; G.L.total[l] = tot + (uint32_t)add - ey; }
      __syncwarp();
      G.tick(ticks);
      return;
    }
    // the values and the added runs (value, count; place, 0) in shared memory
    // where they fit: the searches below are chains of dependent loads
    uint2 *fr = G.tmp;
    const uint32_t *X = &p[0].x;
    uint32_t xs = 2, e = 0;  // e: the removed run's index + 1
    // a few values: each by all lanes, 32 probes a round, without a look at all runs
    const bool few = sn <= 4 && nstage >= 8;
    const bool staged = !few && 2ull * sn + (n + 1) / 2 <= nstage;
    if (few) fr = stage;
    if (staged) {
      fr = stage;
      uint32_t *sx = reinterpret_cast<uint32_t *>(stage + 2 * sn);
#pragma unroll 4
      for (uint32_t i = lane; i < n; i += 32) {
        const uint32_t x = p[i].x;
        sx[i] = x;
        if (x == r) e = i + 1;
      }
      X = sx;
      xs = 1;
      e = __reduce_max_sync(FULL_WARP, e);
      __syncwarp();
    } else {
      if (!few && 2ull * sn > G.tmp_cap) { G.fail = true; return; }
      if (has_r) {
        e = lower(p, n, r);
        e = e < n && p[e].x == r ? e + 1 : 0;
      }
    }
    const bool ex = has_r && e != 0;
    e = ex ? e - 1 : n;
    const uint32_t ey = ex ? p[e].y : 0;
    auto lower_x = [&](uint32_t x) -> uint32_t {
      uint32_t lo = 0, hi = n;
      while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        if (X[m * xs] < x) lo = m + 1; else hi = m;
      }
      return lo;
    };
    uint32_t knew = 0, ebef = 0;  // added runs, and those before the removed one
    unsigned long long ticks = 0, add = 0;
    bool bad = false;
    for (uint32_t q0 = 0; q0 < sn; q0 += 32) {
      const uint32_t q = q0 + lane;
      uint2 s = make_uint2(skip, 0);
      if (q < sn) s = S[q];
      const bool valid = q < sn && s.x != skip;
      const unsigned long long c = (unsigned long long)s.y * mult;
      uint32_t pos = 0;
      bool dup = false;
      if (few)
        for (uint32_t j = 0; j < sn; ++j) {
          const uint32_t at = lower(p, n, __shfl_sync(FULL_WARP, s.x, j));
          if ((uint32_t)lane == j) pos = at;
        }
      if (valid) {
        if (c > 0xffffffffull) bad = true;
        if (!few) pos = lower_x(s.x);
        dup = pos < n && X[pos * xs] == s.x;
        if (dup) {
          const uint32_t y = p[pos].y;
          if (y > 0xffffffffu - (uint32_t)c) bad = true;
          p[pos].y = y + (uint32_t)c;
        } else {
          ticks += n - pos;
        }
        add += c;
        if (mark_a && (dup || c >= 2)) mark(l >> 1, s.x);
      }
      const unsigned b = __ballot_sync(FULL_WARP, valid && !dup);
      if (valid && !dup) {
        const uint32_t o = 2 * (knew + __popc(b & lt()));
        fr[o] = make_uint2(s.x, (uint32_t)c);
        fr[o + 1] = make_uint2(pos, 0);
      }
      knew += __popc(b);
      if (ex) ebef += __popc(__ballot_sync(FULL_WARP, valid && !dup && s.x < r));
    }
    add = warp_sum64(add);
    ticks = warp_sum64(ticks);
    if (mark_a) ticks += add;
    __syncwarp();
    if (__any_sync(FULL_WARP, bad) || tot + add > 0xffffffffull || (unsigned long long)n + knew > 0xffffffffull) {
      G.fail = true;
      return;
    }
    if (ex) ticks += (unsigned long long)(n + knew) - (e + ebef);
    const uint32_t m = n + knew - (ex ? 1u : 0u);
    uint32_t off = off0;
    if (m > cap && !grow(l, cap, m, off)) return;
    uint2 *dst = G.L.pool + off;
    // added runs at or before run i's place
    const uint32_t pos0 = knew ? fr[1].x : n;
    auto shift = [&](uint32_t i) -> uint32_t {
      if (knew <= 1) return i >= pos0 ? knew : 0u;
      uint32_t lo = 0, hi = knew;
      while (lo < hi) {
        const uint32_t c = (lo + hi) >> 1;
        if (fr[2 * c + 1].x <= i) lo = c + 1; else hi = c;
      }
      return lo;
    };
    constexpr int U = 8;  // runs per lane in flight
    const uint32_t first = dst == p ? min(pos0, e) : 0;  // runs before it keep their place
    // runs that move to a higher place, from the back (in a new place: all runs;
    // with one added run for the removed one, those between the two places)
    const uint32_t end = dst != p || knew > 1 || (knew == 1 && !ex) ? n : knew == 1 && pos0 <= e ? e : first;
    for (uint32_t hi = end; hi > first;) {
      const uint32_t lo = hi - first > 32 * U ? hi - 32 * U : first;
      uint2 v[U];
      uint32_t to[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t i = lo + u * 32 + lane;
        to[u] = 0xffffffffu;
        if (i < hi && i != e) {
          v[u] = p[i];
          const uint32_t t = i + shift(i) - (ex && i > e ? 1u : 0u);
          if (dst != p || t > i) to[u] = t;
        }
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (to[u] != 0xffffffffu) dst[to[u]] = v[u];
      __syncwarp();
      hi = lo;
    }
    // runs between the removed one and the first added one move one place down
    if (dst == p && ex && pos0 > e + 1)
      for (uint32_t lo = e + 1; lo < pos0; lo += 32 * U) {
        uint2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t i = lo + u * 32 + lane;
          if (i < pos0) v[u] = p[i];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t i = lo + u * 32 + lane;
          if (i < pos0) p[i - 1] = v[u];
        }
        __syncwarp();
      }
    for (uint32_t q = lane; q < knew; q += 32) {
      const uint32_t pos = fr[2 * q + 1].x;
      dst[pos + q - (ex && e < pos ? 1u : 0u)] = fr[2 * q];
    }
    if (lane == 0) {
      G.L.nrun[l] = m;
      G.L.total[l] = tot + (uint32_t)add - ey;
    }
    __syncwarp();
    G.tick(ticks);
  }

  // One lane's share of a cancellation: list l of n runs (n <= N) takes the
  // value ad (k = 1) with count mult * ad.y and loses r's run.
  template <int N>
  struct LaneEdit {
    uint2 v[N], ad;
    uint32_t apos, m, e;
    bool fresh, bad;
    unsigned long long total, ticks;

    __device__ __forceinline__ void load(const WarpGraph &W, bool on, const uint2 *p, uint32_t n, uint32_t tot,
                                         uint2 add, uint32_t k, uint32_t mult, uint32_t r, bool mark_a, uint32_t self) {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = on && (uint32_t)i < n ? p[i] : make_uint2(0xffffffffu, 0u);
      const bool adds = on && k != 0;
      const unsigned long long c = (unsigned long long)add.y * mult;
      ad = make_uint2(add.x, (uint32_t)c);
      apos = 0;
      bad = adds && c > 0xffffffffull;
      bool dup = false;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        apos += v[i].x < ad.x;
        if (adds && v[i].x == ad.x) {
          dup = true;
          if (c > 0xffffffffull - v[i].y) bad = true;
          v[i].y += (uint32_t)c;
        }
      }
      fresh = adds && !dup;
      m = n + (fresh ? 1u : 0u);
      ticks = fresh ? n - apos : 0u;
      total = tot + (adds ? c : 0ull);
      if (total > 0xffffffffull) bad = true;
      if (mark_a && adds) {
        ticks += c;
        if (dup || c >= 2) W.mark(self, ad.x);
      }
      e = N;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (on && v[i].x == r) { e = i; total -= v[i].y; }
      if (e < N) {
        ticks += m - (e + (fresh && ad.x < r ? 1u : 0u));
        --m;
      }
    }
    __device__ __forceinline__ void store(uint2 *p, uint32_t n) const {
#pragma unroll
      for (int i = 0; i < N; ++i)
        if ((uint32_t)i < n && (uint32_t)i != e) p[i - (e < (uint32_t)i ? 1u : 0u) + (fresh && ad.x < v[i].x ? 1u : 0u)] = v[i];
      if (fresh) p[apos - (e < apos ? 1u : 0u)] = ad;
    }
  };
  // All lanes: the edits of the lanes with `on`; false when the pass failed.
  template <int N>
  __device__ __forceinline__ bool lane_edits(bool on, uint32_t l, uint32_t n, uint32_t cap, uint32_t tot, uint32_t off,
                                             uint2 add, uint32_t k, uint32_t mult, uint32_t r, bool mark_a) {
    LaneEdit<N> E;
    E.load(*this, on, G.L.pool + off, n, tot, add, k, mult, r, mark_a, l >> 1);
    uint32_t room = 0;  // for a list that outgrows its place
    if (on && E.m > cap) {
      room = cap * 2 + 4;
      while (room < E.m) room *= 2;
    }
    if (__any_sync(FULL_WARP, E.bad)) G.fail = true;
    if (__any_sync(FULL_WARP, room != 0)) {
      uint32_t all;
      const uint32_t at = warp_exscan(room, lane, all);
      const unsigned long long base = take_room(all);
      if (!G.fail && room) {
        off = (uint32_t)base + at;
        G.L.off[l] = off;
        G.L.cap[l] = room;
      }
    }
    if (G.fail) return false;
    if (on) {
      E.store(G.L.pool + off, n);
      G.L.nrun[l] = E.m;
      G.L.total[l] = (uint32_t)E.total;
    }
    __syncwarp();
    return G.tick(warp_sum64(on ? E.ticks : 0ull));
  }

  // A pair to cancel: both points' lists' places and lengths (asc, des).
  struct Pair {
    uint2 o0, o1, n0, n1;
    uint32_t cp0, cp1;
  };
  // cp0 becomes the point whose asc list holds the other; false when neither does
  __device__ __forceinline__ bool orient(Pair &q) const {
    if (holds(G.L.pool + q.o0.x, q.n0.x, q.cp1)) return true;
    q = Pair{q.o1, q.o0, q.n1, q.n0, q.cp1, q.cp0};
    return holds(G.L.pool + q.o0.x, q.n0.x, q.cp1);
  }
  // the pair itself: cancelled, des(cp0) and asc(cp1) empty (flags: further flags of both)
  __device__ __forceinline__ void close(const Pair &q, uint8_t flags) const {
    if (lane == 0) {
      G.flags[q.cp0] |= F_CANCELLED | flags;
      G.flags[q.cp1] |= F_CANCELLED | flags;
      G.L.nrun[2 * q.cp0 + 1] = G.L.total[2 * q.cp0 + 1] = 0;
      G.L.nrun[2 * q.cp1] = G.L.total[2 * q.cp1] = 0;
    }
  }
  // The edits of all neighbours' lists, by warp `who` of `warps`: the short
  // lists by warp 0, the longer ones in turn.  Every warp sorts the lists into
  // short and long by their lengths, so none of them is edited before all
  // warps have read its length (barrier BAR_EDIT of those warps, once per 32
  // neighbours: no warp leaves early).
  __device__ __forceinline__ void edit_neighbours(const Pair &q, int who, int warps) {
    const uint32_t cp0 = q.cp0, cp1 = q.cp1;
    const uint2 o0 = q.o0, o1 = q.o1;
    const uint2 *pA = G.L.pool + o0.x, *pD = G.L.pool + o1.y;
    const uint32_t nA = q.n0.x, nE0 = q.n0.y, nE1 = q.n1.x, nD = q.n1.y;
    const uint32_t tD = nA, tE0 = nA + nD, tE1 = tE0 + nE0, nt = tE1 + nE1;
    int turn = 0;  // the warp that took the last longer list
    // The added value of either side where there is at most one (k: how many, 2
    // for more): the list without the other point, from its first two runs.
    uint2 fA[2], fD[2];
#pragma unroll
    for (uint32_t q = 0; q < 2; ++q) {
      fA[q] = q < nA ? pA[q] : make_uint2(cp1, 0);
      fD[q] = q < nD ? pD[q] : make_uint2(cp0, 0);
    }
    const bool a0 = fA[0].x != cp1, a1 = fA[1].x != cp1, d0 = fD[0].x != cp0, d1 = fD[1].x != cp0;
    const uint2 addA = a0 ? fA[0] : fA[1], addD = d0 ? fD[0] : fD[1];
    const uint32_t kA = nA > 2 ? 2u : (a0 ? 1u : 0u) + (a1 ? 1u : 0u), kD = nD > 2 ? 2u : (d0 ? 1u : 0u) + (d1 ? 1u : 0u);
    for (uint32_t t0 = 0; t0 < nt; t0 += 32) {
      const uint32_t t = t0 + lane;
      // side 0: a neighbour a of cp0 (its des list), 1: a neighbour d of cp1
      // (its asc list), 2 / 3: an erase from an asc / a des list only
      int side = t < tD ? 0 : t < tE0 ? 1 : t < tE1 ? 2 : t < nt ? 3 : -1;
      const uint32_t at = side == 0 ? o0.x + t : side == 1 ? o1.y + (t - tD) : side == 2 ? o0.y + (t - tE0) : o1.x + (t - tE1);
      uint2 v = make_uint2(0, 0);
      if (side >= 0) v = G.L.pool[at];
      if ((side == 0 && v.x == cp1) || (side == 1 && v.x == cp0)) side = -1;
      const uint32_t l = 2 * v.x + (side == 0 || side == 3 ? 1u : 0u), mult = v.y, r = side == 0 || side == 2 ? cp0 : cp1;
      const uint32_t ka = side == 0 ? kD : side == 1 ? kA : 0;
      uint32_t n = 0, cap = 0, tot = 0, off = 0;
      if (side >= 0) { n = G.L.nrun[l]; cap = G.L.cap[l]; tot = G.L.total[l]; off = G.L.off[l]; }
      const uint2 ad = side == 0 ? addD : addA;
      const bool small = side >= 0 && n <= 8 && ka <= 1;
      if (warps > 1) {
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(BAR_EDIT), "r"(32 * warps) : "memory");
      }
      if (G.fail) continue;
      // the long lists' first lines on their way into L1
      if (side >= 0 && n > 256)
        for (uint32_t q = 0; q < 256; q += 16) asm volatile("prefetch.global.L1 [%0];" ::"l"(G.L.pool + off + q));
      // (mostly a saddle's neighbours or an extremum's saddles: two runs, one added value)
      if (who == 0) {
        if (!__any_sync(FULL_WARP, small && n > 4)) lane_edits<4>(small, l, n, cap, tot, off, ad, ka, mult, r, side == 0);
        else lane_edits<8>(small, l, n, cap, tot, off, ad, ka, mult, r, side == 0);
      }
      // the longer lists, each by all lanes of a warp; they go round from the warp
      // after the last one that took one (warp 0 last: it has the short lists)
      unsigned big = __ballot_sync(FULL_WARP, side >= 0 && !small);
      const int nbig = __popc(big);
      int wait = (who + 2 * warps - turn - 1) % warps;  // lists before this warp's first
      turn = (turn + nbig) % warps;
      if (wait >= nbig) continue;
      for (; big && !G.fail; big &= big - 1) {
        if (wait-- != 0) continue;
        wait = warps - 1;
        const int s = __ffs(big) - 1;
        const int bs = __shfl_sync(FULL_WARP, side, s);
        const uint32_t bl = __shfl_sync(FULL_WARP, l, s), bm = __shfl_sync(FULL_WARP, mult, s);
        uint32_t bn = __shfl_sync(FULL_WARP, n, s), bc = __shfl_sync(FULL_WARP, cap, s);
        uint32_t bt = __shfl_sync(FULL_WARP, tot, s), bo = __shfl_sync(FULL_WARP, off, s);
        const uint2 *S = bs == 0 ? pD : pA;
        uint32_t sn = bs == 0 ? nD : bs == 1 ? nA : 0u;
        // more added values than the scratch holds: ascending parts, one merge each
        for (const uint32_t part = (uint32_t)min(G.tmp_cap / 2, 1ull << 30); sn > part && sn > 32 && !G.fail; sn -= part, S += part) {
          edit_list(bl, bn, bc, bt, bo, S, part, bs == 0 ? cp0 : cp1, bm, false, 0u, bs == 0);
          bn = G.L.nrun[bl]; bc = G.L.cap[bl]; bt = G.L.total[bl]; bo = G.L.off[bl];
        }
        if (!G.fail)
          edit_list(bl, bn, bc, bt, bo, S, sn, bs == 0 ? cp0 : cp1, bm, true, bs == 0 || bs == 2 ? cp0 : cp1, bs == 0);
      }
    }
  }

  // List l := the multiset of the items of the first n lanes, in any order
  // (the other lanes: a value above every index, count 0).
  __device__ __forceinline__ bool set_list_lanes(uint32_t l, uint2 v, uint32_t n, uint32_t cap) {
    uint32_t before = __shfl_up_sync(FULL_WARP, v.x, 1);
    if (__any_sync(FULL_WARP, lane > 0 && v.x < before)) {
      for (uint32_t k = 2; k < 2 * n; k <<= 1)  // bitonic
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
          const uint32_t ox = __shfl_xor_sync(FULL_WARP, v.x, j), oy = __shfl_xor_sync(FULL_WARP, v.y, j);
          const bool low = ((lane & j) == 0) == ((lane & k) == 0);
          if (low ? ox < v.x : ox > v.x) v = make_uint2(ox, oy);
        }
      before = __shfl_up_sync(FULL_WARP, v.x, 1);
    }
    const bool head = (uint32_t)lane < n && (lane == 0 || v.x != before);
    const unsigned hm = __ballot_sync(FULL_WARP, head);
    const uint32_t m = __popc(hm);
    unsigned long long sum = v.y;
    if (m != n)  // equal neighbours become one run
      for (uint32_t q = 1; q < n; ++q) {
        const uint32_t ox = __shfl_down_sync(FULL_WARP, v.x, q), oy = __shfl_down_sync(FULL_WARP, v.y, q);
        if (lane + q < n && ox == v.x) sum += oy;
      }
    const unsigned long long tot = warp_sum64(head ? sum : 0ull);
    if (__any_sync(FULL_WARP, head && sum > 0xffffffffull) || tot > 0xffffffffull) { G.fail = true; return false; }
    uint32_t off = G.L.off[l];
    if (m > cap && !grow(l, cap, m, off)) return false;
    if (head) G.L.pool[off + __popc(hm & lt())] = make_uint2(v.x, (uint32_t)sum);
    if (lane == 0) { G.L.nrun[l] = m; G.L.total[l] = (uint32_t)tot; }
    __syncwarp();
    return true;
  }

  // List l := the multiset of the n (value, count) items of b in any order
  // (b: the stage or the graph's scratch runs).
  __device__ __forceinline__ bool set_list(uint32_t l, uint2 *b, unsigned long long n) {
    if (!G.tick(n + 1)) return false;
    const uint32_t cap = G.L.cap[l];
    if (n <= 32) {  // in registers
      uint2 v = make_uint2(0xffffffffu, 0u);
      if ((unsigned)lane < n) v = b[lane];
      return set_list_lanes(l, v, (uint32_t)n, cap);
    }
    const unsigned long long room = b == stage ? nstage : b == shared_stage ? nshared_stage : G.tmp_cap;
    unsigned long long N = 64;
    while (N < n) N <<= 1;
    if (N <= room) {  // bitonic, padded to a power of two by values above every index
      for (unsigned long long i = n + lane; i < N; i += 32) b[i] = make_uint2(0xffffffffu, 0u);
      __syncwarp();
      const bool counts = lane == 0 && N >= 4096;
      for (unsigned long long k = 2; k <= N; k <<= 1)
        for (unsigned long long j = k >> 1; j > 0; j >>= 1) {
          if (counts) moved_on();
          for (unsigned long long t = lane; t < N / 2;) {
            const unsigned long long end = min(t + 32 * BEAT_STEPS, N / 2);
#pragma unroll 4
            for (; t < end; t += 32) {
              const unsigned long long i = 2 * t - (t & (j - 1)), o = i + j;  // the t-th pair at distance j
              const uint2 x = b[i], y = b[o];
              if ((x.x > y.x) == ((i & k) == 0)) { b[i] = y; b[o] = x; }
            }
            if (counts) moved_on();
          }
          __syncwarp();
        }
    } else {
      if (lane == 0) {  // heap sort, as Graph::sort_tmp
        for (unsigned long long s = n / 2; s-- > 0;) {
          if ((s & 1023) == 0) moved_on();
          G.sift(s, n);
        }
        for (unsigned long long e = n; e-- > 1;) {
          if ((e & 1023) == 0) moved_on();
          const uint2 q = b[0];
          b[0] = b[e];
          b[e] = q;
          G.sift(0, e);
        }
      }
      __syncwarp();
    }
    // equal neighbours become one run
    auto is_head = [&](unsigned long long u) { return u < n && (u == 0 || b[u - 1].x != b[u].x); };
    uint32_t m = 0;
    for (unsigned long long u0 = 0; u0 < n; u0 += 32) {
      if (lane == 0 && ((u0 + 32) & (32 * BEAT_STEPS - 1)) == 0) moved_on();
      m += __popc(__ballot_sync(FULL_WARP, is_head(u0 + lane)));
    }
    uint32_t off = G.L.off[l];
    if (m > cap && !grow(l, cap, m, off)) return false;
    uint2 *p = G.L.pool + off;
    unsigned long long tot = 0;
    bool bad = false;
    uint32_t w = 0;
    for (unsigned long long u0 = 0; u0 < n; u0 += 32) {
      if (lane == 0 && ((u0 + 32) & (32 * BEAT_STEPS - 1)) == 0) moved_on();
      const unsigned long long u = u0 + lane;
      const bool head = is_head(u);
      const unsigned hb = __ballot_sync(FULL_WARP, head);
      if (head) {
        const uint32_t x = b[u].x;
        unsigned long long s = 0;
        for (unsigned long long q = u; q < n && b[q].x == x;) {
          const unsigned long long end = min(q + BEAT_STEPS, n);
          for (; q < end && b[q].x == x; ++q) s += b[q].y;
          if (q >= u + BEAT_STEPS) moved_on();
        }
        if (s > 0xffffffffull) bad = true;
        tot += s;
        p[w + __popc(hb & lt())] = make_uint2(x, (uint32_t)s);
      }
      w += __popc(hb);
    }
    tot = warp_sum64(tot);
    if (__any_sync(FULL_WARP, bad) || tot > 0xffffffffull) { G.fail = true; return false; }
    if (lane == 0) { G.L.nrun[l] = m; G.L.total[l] = (uint32_t)tot; }
    __syncwarp();
    return true;
  }
  // a new place for list l, whose runs are all rewritten
  __device__ __forceinline__ bool grow(uint32_t l, uint32_t cap, uint32_t m, uint32_t &off) {
    uint32_t nc = cap * 2 + 4;
    while (nc < m) nc *= 2;
    const unsigned long long at = take_room(nc);
    if (G.fail) return false;
    off = (uint32_t)at;
    if (lane == 0) { G.L.off[l] = off; G.L.cap[l] = nc; }
    return true;
  }
  // n runs at the top of the pool (shared by the team's warps, or by all blocks)
  __device__ __forceinline__ unsigned long long take_room(unsigned long long n) {
    unsigned long long at = G.L.top;
    if (team) {
      if (lane == 0) at = team->shared_top ? atomicAdd(team->shared_top, n) : atomicAdd(&team->top, n);
      at = __shfl_sync(FULL_WARP, at, 0);
    }
    if (at + n > G.L.pool_cap) G.fail = true;
    else G.L.top = at + n;
    return at;
  }

  // A run of the list that uncancel_pairs rewrites, one per lane: a surviving
  // neighbour stays, a cancelled pair's saddle or extremum gives way to its
  // partner's list (open: cnt runs at src), the pair's other point goes (cnt 0).
  struct Item {
    uint2 run;
    uint32_t cnt, src;
    bool open, wrong, stopped;
  };
  __device__ __forceinline__ Item item_of(const uint2 *p, uint32_t nr, uint32_t k, uint32_t other, int i, uint32_t turn) const {
    Item t{make_uint2(other, 0), 0, 0, false, false, false};
    if (k < nr) t.run = p[k];
    const uint32_t x = t.run.x;
    if (x != other) {
      const uint8_t f = G.flags[x];
      t.cnt = 1;
      if (f & F_BCANCEL) {
        const uint32_t q = G.pair_idx[x];
        bool cancelled = f & F_CANCELLED;
        const bool back = q < G.ncp && G.pair_idx[q] == x;
        if (ord) {  // x's pair, if it is one of the pass: later on the list, or still cancelled at this one's turn
          const uint32_t o = ord[x];
          if (o) {
            cancelled = o <= turn;
            const uint32_t bit = 2 * (o - 1) + i;
            volatile const uint32_t *w = done + (bit >> 5);
            for (unsigned long long polls = 0; !cancelled && !((*w >> (bit & 31)) & 1u);)
              if (++polls > WAIT_LIMIT || called_off()) {
                t.stopped = true;  // the polls ran out, or another warp's pair failed
                break;
              }
            __threadfence_block();
          }
        }
        if (cancelled || !back) {
          t.wrong = true;
          t.cnt = 0;
        } else {
          t.open = true;
          t.cnt = G.L.nrun[2 * q + i];
          t.src = G.L.off[2 * q + i];
        }
      }
    }
    return t;
  }
  // The lanes' items into b, a short list by its lane, a longer one by all lanes; their number.
  __device__ __forceinline__ uint32_t put_items(const Item &t, uint2 *b, bool &wrong, bool &bad) const {
    uint32_t all;
    const uint32_t o = warp_exscan(t.cnt, lane, all);
    if (t.cnt && !t.open) b[o] = t.run;
    auto one = [&](uint2 v, uint32_t y, uint32_t to) {
      if (G.flags[v.x] & F_BCANCEL) wrong = true;
      const unsigned long long c = (unsigned long long)y * v.y;
      if (c > 0xffffffffull) bad = true;
      b[to] = make_uint2(v.x, (uint32_t)c);
    };
    if (t.open && t.cnt <= 2) {
      if (t.cnt > 0) one(G.L.pool[t.src], t.run.y, o);
      if (t.cnt > 1) one(G.L.pool[t.src + 1], t.run.y, o + 1);
    }
    for (unsigned lg = __ballot_sync(FULL_WARP, t.open && t.cnt > 2); lg; lg &= lg - 1) {
      const int s = __ffs(lg) - 1;
      const uint32_t sc = __shfl_sync(FULL_WARP, t.cnt, s), ss = __shfl_sync(FULL_WARP, t.src, s);
      const uint32_t so = __shfl_sync(FULL_WARP, o, s), sy = __shfl_sync(FULL_WARP, t.run.y, s);
      for (uint32_t q = lane; q < sc; q += 32) {
        if (((q + 32) & (32 * BEAT_STEPS - 1)) == 0) moved_on();  // (lane 0)
        one(G.L.pool[ss + q], sy, so + q);
      }
    }
    return all;
  }

  // The scratch for n items: the warp's own where they fit, else one that the
  // team's warps share and hold one at a time (drop_scratch), else the
  // graph's; null when the pass failed.
  __device__ __forceinline__ uint2 *take_scratch(unsigned long long n) {
    if (stage && n <= nstage) return stage;
    if (team) {
      bool got = false;
      for (unsigned long long seen = ~0ull;;) {
        if (lane == 0)
          for (unsigned long long polls = 0; !got && polls <= WAIT_LIMIT; ++polls) {
            got = atomicCAS(&team->lock, 0, 1) == 0;
            if (!got && called_off()) break;
          }
        got = __shfl_sync(FULL_WARP, got, 0);
        if (got || !wait_on(seen)) break;
      }
      __threadfence_block();
      if (!got) { G.fail = true; return nullptr; }
    }
    if (shared_stage && n <= nshared_stage) return shared_stage;
    if (n > G.tmp_cap) { drop_scratch(n); G.fail = true; return nullptr; }
    return G.tmp;
  }
  __device__ __forceinline__ void drop_scratch(unsigned long long n) {
    __syncwarp();
    if (team && n > nstage && lane == 0) {
      __threadfence_block();
      atomicExch(&team->lock, 0);
    }
  }

  // uncancel_pairs (see Graph::uncancel_pairs): false on a reference logic_error condition
  __device__ __forceinline__ bool uncancel_pairs(uint32_t c1, uint32_t c2) {
    if (!holds(G.runs(2 * c1), G.L.nrun[2 * c1], c2)) { const uint32_t t = c1; c1 = c2; c2 = t; }
    for (int i = 0; i < 2; ++i) {
      if (!uncancel_list(c1, c2, i, 0)) return false;
      if (G.fail) return true;
    }
    if (lane == 0) {
      G.flags[c1] &= ~F_CANCELLED;
      G.flags[c2] &= ~F_CANCELLED;
    }
    __syncwarp();
    return true;
  }
  // Its part that rewrites asc(c1) (i = 0) or des(c2) (i = 1).  turn: 1 + the
  // pair's place on the cancellation list (side by side only).
  __device__ __forceinline__ bool uncancel_list(uint32_t c1, uint32_t c2, int i, uint32_t turn) {
    const uint32_t l = i ? 2 * c2 + 1 : 2 * c1, other = i ? c1 : c2;
    uint2 *p = G.runs(l);
    const uint32_t nr = G.L.nrun[l];
    bool wrong = false, bad = false;
    unsigned long long n = 0, ticks = 0;
    uint2 *b;
    if (nr <= 32) {  // one run per lane
      Item t;
      for (unsigned long long seen = ~0ull;;) {
        t = item_of(p, nr, lane, other, i, turn);
        if (!__any_sync(FULL_WARP, t.stopped)) break;
        if (!wait_on(seen)) { G.fail = true; return true; }
      }
      if (!__any_sync(FULL_WARP, (uint32_t)lane < nr && t.run.x == other)) return false;  // "cancellable pair is not connected"
      if (__any_sync(FULL_WARP, t.wrong)) return false;
      if (!__any_sync(FULL_WARP, t.open)) {  // the list without the other point
        const unsigned keep = __ballot_sync(FULL_WARP, t.cnt != 0);
        const unsigned long long tot = warp_sum64(t.cnt ? t.run.y : 0ull);
        n = __popc(keep);
        if (!G.tick(n + 1)) return true;
        if (tot > 0xffffffffull) { G.fail = true; return true; }
        if (t.cnt) p[__popc(keep & lt())] = t.run;
        if (lane == 0) { G.L.nrun[l] = (uint32_t)n; G.L.total[l] = (uint32_t)tot; }
        __syncwarp();
        return true;
      }
      n = warp_sum64(t.cnt);
      ticks = warp_sum64(t.open ? 1ull + t.cnt : 0ull);
      if (!(b = take_scratch(n))) return true;
      put_items(t, b, wrong, bad);
    } else {
      if (!holds(p, nr, other)) return false;
      for (uint32_t k0 = 0; k0 < nr; k0 += 32) {  // the items' number, and the checks
        if (lane == 0 && ((k0 + 32) & (32 * BEAT_STEPS - 1)) == 0) moved_on();
        Item t;
        for (unsigned long long seen = ~0ull;;) {
          t = item_of(p, nr, k0 + lane, other, i, turn);
          if (!__any_sync(FULL_WARP, t.stopped)) break;
          if (!wait_on(seen)) { G.fail = true; return true; }
        }
        wrong |= t.wrong;
        n += warp_sum64(t.cnt);
        ticks += warp_sum64(t.open ? 1ull + t.cnt : 0ull);
      }
      if (__any_sync(FULL_WARP, wrong)) return false;
      if (!(b = take_scratch(n))) return true;
      uint2 *to = b;
      for (uint32_t k0 = 0; k0 < nr; k0 += 32) to += put_items(item_of(p, nr, k0 + lane, other, i, turn), to, wrong, bad);
    }
    __syncwarp();
    if (__any_sync(FULL_WARP, bad)) G.fail = true;
    const bool off = __any_sync(FULL_WARP, wrong);
    if (!off && !G.fail && G.tick(ticks)) set_list(l, b, n);
    drop_scratch(n);
    return !off;
  }

  // A warp's share of uncancelling the pairs canc[0..npairs) (first the point
  // whose asc list holds the other), the last one first, asc and des list as
  // tasks of their own, taken in order from team->ticket (2 * npairs at the
  // start).  `ord` and `done` are set up for them; the CANCELLED flags stay.
  __device__ __forceinline__ void uncancel_shared(const uint2 *canc, uint32_t npairs) {
    for (;;) {
      unsigned long long t = 0;
      if (lane == 0) t = atomicAdd(&team->ticket, ~0ull);  // takes one
      t = __shfl_sync(FULL_WARP, t, 0);
      if (t == 0 || t > 2ull * npairs) break;  // none left
      if (__any_sync(FULL_WARP, *(volatile uint32_t *)&team->fail || *(volatile uint32_t *)&team->wrong)) break;
      const uint32_t k = (uint32_t)((t - 1) / 2), i = (uint32_t)(t & 1);
      const uint2 c = canc[k];
      if (!uncancel_list(c.x, c.y, (int)i, k + 1)) team->wrong = 1;
      if (G.fail) {
        team->fail = 1;
        break;
      }
      __threadfence_block();
      __syncwarp();
      if (lane == 0) atomicOr(&done[(2 * k + i) >> 5], 1u << ((2 * k + i) & 31));
    }
  }
};

}  // namespace dmsc
