// sort.cu -- stable LSD radix sort of (key, value) pairs of 32-bit words
// (the reference's sort slot: BitonicSortProgram, dmsc/include/bitonic_sort.h).
//
// The scheme is the published single-pass one (Adinets and Merrill, "Onesweep",
// 2022, after Merrill and Garland's decoupled look-back, 2016).  One pass over
// the keys counts the digits of all passes.  Each pass then takes the pairs
// once: a block ranks a tile's pairs by their digit, learns
// how many pairs of each digit the earlier tiles hold by decoupled look-back
// (tiles are taken from an atomic counter, so a block only waits for blocks
// that already run), groups the tile by digit in shared memory, and writes
// every group as one contiguous piece.  Memory bounds it, 16 bytes a pair and
// pass, and with it the look-back, whose traffic goes with the square of the
// tiles in flight (256 words for each tile before a tile): for many pairs a tile
// is as large as one block's registers and shared memory allow, one block per SM.
// With 6,144 pairs a tile a pass over 3,000,017 took 41 us, with 20,480 31; a
// histogram, a scan and a scatter of single pairs took 75 (a warp's 32 pairs
// went to 32 places).  Such tiles leave SMs idle and are long for fewer pairs: up to
// 1.6 million the tiles have 4,096 (a call with 130,000 pairs 158 us with 20,480 a
// tile, 90 so; 900,000: 165, 125; 1,500,000: 169, 154; they meet near 2 million, and
// the line lies below, where the smaller tiles still gain a tenth).  Up to 8,192 pairs are
// sorted by one block in one launch, 4 or 8 a thread (a call with 3,000 pairs 104
// us with 20 a thread, 51 so; 6,000: 104, 61).
#include "dmsc_common.cuh"
#include "dmsc_internal.h"
#include "smem_limit.h"

#include <algorithm>

namespace dmsc {

namespace {

constexpr int RS_THREADS = 1024, RS_WARPS = RS_THREADS / 32;
// pairs per thread; each warp owns a contiguous run of 32 times as many, a tile
// has RS_THREADS times as many
constexpr int RS_ITEMS = 20, RS_FEW = 4, RS_SMALL = 8;
constexpr long long RS_FEW_MAX = 400ll * RS_THREADS * RS_FEW;
// pairs of the tiles that n pairs are cut into (n of them: one launch)
constexpr long long radix_tile(long long n) {
  return RS_THREADS * (n <= RS_THREADS * RS_SMALL ? RS_SMALL : n <= RS_FEW_MAX ? RS_FEW : RS_ITEMS);
}
constexpr int RS_LOOK = 8;                      // earlier tiles looked at together
constexpr int RS_MAX_PASSES = 8;                // 4 digits of the key, up to 4 of the array number
constexpr unsigned long long RS_LIMIT = 1ull << 22;  // polls of an earlier tile's word

template <int ITEMS>
struct RadixSmem {
  uint32_t key[RS_THREADS * ITEMS], val[RS_THREADS * ITEMS];
  uint16_t cnt[RS_WARPS][256];  // per warp and digit: pairs, then the pairs of the warps before it
  uint32_t first[256];          // the digit's first place in the tile
  uint32_t to[256];             // a pair's place in the output, less its place in the tile
  uint32_t wsum[8];
  uint32_t tile, late;
};
static_assert(RS_THREADS * RS_ITEMS < 65536, "places in a tile fit 16 bits");

// One pass: digit = (key >> shift) & 255, or with len the digit of the value's
// array number (value / len; the value is then the pair's original index).
struct RadixPass {
  const uint32_t *kin, *vin;  // vin null: the value is the pair's index
  uint32_t *kout, *vout;
  const uint32_t *gather;     // the values written are gather[value]
  uint32_t xin, xout;         // the keys are complemented on the way in / out
  int shift;
  uint32_t len;
};
template <bool ARRAY>
__device__ __forceinline__ uint32_t digit_of(uint32_t key, uint32_t val, int shift, uint32_t len) {
  return ((ARRAY ? val / len : key) >> shift) & 255u;
}

// A tile's pairs: loaded, ranked by digit, and grouped in S.key / S.val in
// stable order; S.first has each digit's first place.  Returns, for threads
// below 256, the tile's pairs of digit threadIdx.x.
template <bool ARRAY, int ITEMS>
__device__ __forceinline__ uint32_t group_tile(RadixSmem<ITEMS> &S, const RadixPass &P, long long base0, long long n, bool from_smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (int k = threadIdx.x; k < RS_WARPS * 128; k += RS_THREADS) reinterpret_cast<uint32_t *>(&S.cnt[0][0])[k] = 0;
  const long long base = base0 + warp * (32 * ITEMS) + lane;
  const int left = (int)(n - base < 32 * ITEMS ? n - base : 32 * ITEMS);  // pairs r * 32 < left are in range
  uint32_t key[ITEMS], val[ITEMS];
  uint16_t rank[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    key[r] = val[r] = 0;
    if (r * 32 < left) {
      const long long i = base + r * 32;
      if (from_smem) {
        key[r] = S.key[i];
        val[r] = S.val[i];
      } else {
        key[r] = P.kin[i] ^ P.xin;
        if (ARRAY) val[r] = P.vin ? P.vin[i] : (uint32_t)i;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const bool valid = r * 32 < left;
    const uint32_t d = digit_of<ARRAY>(key[r], val[r], P.shift, P.len);
    uint32_t peers = __ballot_sync(0xffffffffu, valid);  // the lanes with the same digit
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool on = (d >> b) & 1u;
      const uint32_t v = __ballot_sync(0xffffffffu, on);
      peers &= on ? v : ~v;
    }
    const uint32_t before = S.cnt[warp][d];
    rank[r] = (uint16_t)(before + __popc(peers & lt));
    __syncwarp();
    if (valid && (peers & lt) == 0) S.cnt[warp][d] = (uint16_t)(before + __popc(peers));
    __syncwarp();
  }
  if (!ARRAY && !from_smem) {  // the values, while the digits are summed
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
      if (r * 32 < left) val[r] = P.vin ? P.vin[base + r * 32] : (uint32_t)(base + r * 32);
  }
  __syncthreads();
  uint32_t total = 0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const uint32_t t = S.cnt[w][threadIdx.x];
      S.cnt[w][threadIdx.x] = (uint16_t)total;
      total += t;
    }
    uint32_t x = total;  // the digits' first places
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) S.wsum[warp] = x;
    S.first[threadIdx.x] = x - total;
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    uint32_t b = 0;
    for (int w = 0; w < warp; ++w) b += S.wsum[w];
    S.first[threadIdx.x] += b;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    if (r * 32 >= left) continue;
    const uint32_t d = digit_of<ARRAY>(key[r], val[r], P.shift, P.len), p = S.first[d] + S.cnt[warp][d] + rank[r];
    S.key[p] = key[r];
    S.val[p] = val[r];
  }
  return total;
}

struct RadixShifts {
  int n;
  int shift[RS_MAX_PASSES];
  uint32_t len[RS_MAX_PASSES];
};

// the digits' counts of every pass: hist[256 * pass + digit]
template <int KEYS>  // passes by the key's digits 0 .. KEYS - 1; those of the array number follow
__global__ void __launch_bounds__(1024) k_radix_hist(const uint32_t *__restrict__ keys, uint32_t xin, long long n, RadixShifts P,
                                                     uint32_t *__restrict__ hist) {
  __shared__ uint32_t cnt[RS_MAX_PASSES * 256];
  for (int k = threadIdx.x; k < P.n * 256; k += blockDim.x) cnt[k] = 0;
  __syncthreads();
  constexpr int U = 4;
  const long long step = (long long)gridDim.x * blockDim.x * U;
  for (long long b = (long long)blockIdx.x * blockDim.x * U + threadIdx.x; b < n; b += step) {
    uint32_t k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) k[u] = b + u * blockDim.x < n ? keys[b + u * blockDim.x] ^ xin : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + u * blockDim.x;
      if (i >= n) continue;
#pragma unroll
      for (int p = 0; p < KEYS; ++p) atomicAdd(&cnt[p * 256 + ((k[u] >> (8 * p)) & 255u)], 1u);
      for (int p = KEYS; p < P.n; ++p) atomicAdd(&cnt[p * 256 + digit_of<true>(0, (uint32_t)i, P.shift[p], P.len[p])], 1u);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < P.n * 256; k += blockDim.x)
    if (cnt[k]) atomicAdd(&hist[k], cnt[k]);
}

// word[256 * tile + digit] of a pass: (flag in the top bits, pairs of the digit), flag
// 0 not yet, 1 in the tile, 2 in the tile and all before it; W is 32 bits wide
// below 2^30 pairs.
template <bool ARRAY, typename W, int ITEMS>
__global__ void __launch_bounds__(RS_THREADS, 1) k_radix_pass(RadixPass P, long long n, const uint32_t *__restrict__ hist,
                                                              W *__restrict__ word, uint32_t *__restrict__ counter) {
  constexpr int FLAG = sizeof(W) == 4 ? 30 : 32;
  constexpr W COUNT = ((W)1 << FLAG) - 1;
  extern __shared__ __align__(16) unsigned char radix_smem[];
  constexpr int TILE = RS_THREADS * ITEMS;
  RadixSmem<ITEMS> &S = *reinterpret_cast<RadixSmem<ITEMS> *>(radix_smem);
  if (threadIdx.x == 0) {
    S.tile = atomicAdd(counter, 1u);
    S.late = 0;
  }
  __syncthreads();
  const long long tile = S.tile, base = tile * TILE;
  if (base >= n) return;  // (block-uniform)
  const uint32_t mine = group_tile<ARRAY, ITEMS>(S, P, base, n, false);
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  uint32_t excl = 0;
  if (d < 256) {
    volatile W *w = word + d;
    w[256 * tile] = ((W)(tile ? 1 : 2) << FLAG) | mine;
    unsigned long long polls = 0;
    for (long long j = tile - 1; j >= 0;) {  // RS_LOOK earlier tiles at a time
      W v[RS_LOOK];
#pragma unroll
      for (int q = 0; q < RS_LOOK; ++q) v[q] = j - q >= 0 ? w[256 * (j - q)] : (W)2 << FLAG;
      bool end = false;
#pragma unroll
      for (int q = 0; q < RS_LOOK; ++q) {
        if (end || (v[q] >> FLAG) == 0) { end = true; continue; }
        excl += (uint32_t)(v[q] & COUNT);
        --j;
        if ((v[q] >> FLAG) == 2) { end = true; j = -1; }
      }
      if (j >= 0 && ++polls > RS_LIMIT) { S.late = 1; break; }
    }
  }
  __syncthreads();
  if (S.late) {  // a bounded wait ran out: the earlier tiles' digits counted from their pairs
    uint32_t *c = reinterpret_cast<uint32_t *>(&S.cnt[0][0]);
    for (int k = threadIdx.x; k < 256; k += RS_THREADS) c[k] = 0;
    __syncthreads();
    for (long long i = threadIdx.x; i < base; i += RS_THREADS)
      atomicAdd(&c[digit_of<ARRAY>(P.kin[i] ^ P.xin, P.vin ? P.vin[i] : (uint32_t)i, P.shift, P.len)], 1u);
    __syncthreads();
    if (d < 256) excl = c[d];
  }
  // the digit's first place in the output: the pairs of smaller digits, then those of earlier tiles
  uint32_t h = 0, x = 0;
  if (d < 256) {
    volatile W *w = word + d;
    if (tile) w[256 * tile] = ((W)2 << FLAG) | (W)(excl + mine);
    h = x = hist[d];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) S.wsum[warp] = x;
  }
  __syncthreads();
  if (d < 256) {
    uint32_t b = x - h;
    for (int k = 0; k < warp; ++k) b += S.wsum[k];
    S.to[d] = b + excl - S.first[d];
  }
  __syncthreads();
  const int m = (int)(n - base < TILE ? n - base : TILE);
#pragma unroll 4
  for (int i = threadIdx.x; i < m; i += RS_THREADS) {
    const uint32_t key = S.key[i], val = S.val[i], p = S.to[digit_of<ARRAY>(key, val, P.shift, P.len)] + i;
    P.kout[p] = key ^ P.xout;
    P.vout[p] = P.gather ? P.gather[val] : val;
  }
}

// up to one tile: all passes in one block
template <int ITEMS>
__global__ void __launch_bounds__(RS_THREADS, 1) k_radix_small(RadixPass P, int n, RadixShifts sh) {
  extern __shared__ __align__(16) unsigned char radix_smem[];
  RadixSmem<ITEMS> &S = *reinterpret_cast<RadixSmem<ITEMS> *>(radix_smem);
  for (int p = 0; p < sh.n; ++p) {
    P.shift = sh.shift[p];
    P.len = sh.len[p];
    if (P.len) group_tile<true, ITEMS>(S, P, 0, n, p > 0);
    else group_tile<false, ITEMS>(S, P, 0, n, p > 0);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += RS_THREADS) {
    P.kout[i] = S.key[i] ^ P.xout;
    P.vout[i] = P.gather ? P.gather[S.val[i]] : S.val[i];
  }
}

template <int ITEMS>
cudaError_t radix_run_small(const RadixPass &io, long long n, const RadixShifts &sh, cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = limit.raise(sizeof(RadixSmem<ITEMS>), k_radix_small<ITEMS>);
  if (e != cudaSuccess) return e;
  k_radix_small<ITEMS><<<1, RS_THREADS, sizeof(RadixSmem<ITEMS>), st>>>(io, (int)n, sh);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

// The passes `sh` from (kin, vin) to (kout, vout); the pairs in between go
// through t0 and t1 (keys, then values, n words each; t1 only with more than
// two passes).  The output may be the input.
template <int ITEMS>
cudaError_t radix_run_tiles(const RadixPass &io, long long n, const RadixShifts &sh, uint32_t *const t0[2], uint32_t *const t1[2],
                      cudaStream_t st) {
  constexpr int TILE = RS_THREADS * ITEMS;
  static SmemLimit limit;
  cudaError_t e = limit.raise(sizeof(RadixSmem<ITEMS>), k_radix_pass<false, uint32_t, ITEMS>, k_radix_pass<true, uint32_t, ITEMS>,
                              k_radix_pass<false, unsigned long long, ITEMS>, k_radix_pass<true, unsigned long long, ITEMS>);
  if (e != cudaSuccess) return e;
  const long long nt = (n + TILE - 1) / TILE;
  const bool wide = n >= (1ll << 30);
  const size_t words = 256 * (size_t)nt, head = sizeof(uint32_t) * (256 * RS_MAX_PASSES + 2 * RS_MAX_PASSES);
  const size_t wbytes = (wide ? 8 : 4) * words;
  char *buf = nullptr;  // digit counts and tile counters of the passes, then their words
  e = cudaMallocAsync((void **)&buf, head + wbytes * sh.n, st);
  if (e != cudaSuccess) return e;
  uint32_t *hist = (uint32_t *)buf, *counter = hist + 256 * RS_MAX_PASSES;
  e = cudaMemsetAsync(buf, 0, head + wbytes * sh.n, st);
  int keys = 0;
  while (keys < sh.n && sh.len[keys] == 0) ++keys;
  if (e == cudaSuccess) {
    const unsigned g = (unsigned)std::min<long long>((n + 8191) / 8192, 152 * 2);
    if (keys == 1) k_radix_hist<1><<<g, 1024, 0, st>>>(io.kin, io.xin, n, sh, hist);
    else if (keys == 2) k_radix_hist<2><<<g, 1024, 0, st>>>(io.kin, io.xin, n, sh, hist);
    else if (keys == 3) k_radix_hist<3><<<g, 1024, 0, st>>>(io.kin, io.xin, n, sh, hist);
    else k_radix_hist<4><<<g, 1024, 0, st>>>(io.kin, io.xin, n, sh, hist);
    DMSC_LAUNCHED(1);
    e = cudaGetLastError();
  }
  const uint32_t *k = io.kin, *v = io.vin;
  for (int p = 0; p < sh.n && e == cudaSuccess; ++p) {
    RadixPass q = io;
    q.kin = k;
    q.vin = v;
    q.shift = sh.shift[p];
    q.len = sh.len[p];
    if (p) q.xin = 0;
    if (p + 1 < sh.n) {
      q.kout = (p & 1 ? t1 : t0)[0];
      q.vout = (p & 1 ? t1 : t0)[1];
      q.xout = 0;
      q.gather = nullptr;
    }
    auto go = [&](auto kernel, auto *w) {
      kernel<<<(unsigned)nt, RS_THREADS, sizeof(RadixSmem<ITEMS>), st>>>(q, n, hist + 256 * p, w + words * p, counter + p);
    };
    uint32_t *w4 = (uint32_t *)(buf + head);
    unsigned long long *w8 = (unsigned long long *)(buf + head);
    if (wide) q.len ? go(k_radix_pass<true, unsigned long long, ITEMS>, w8) : go(k_radix_pass<false, unsigned long long, ITEMS>, w8);
    else q.len ? go(k_radix_pass<true, uint32_t, ITEMS>, w4) : go(k_radix_pass<false, uint32_t, ITEMS>, w4);
    DMSC_LAUNCHED(1);
    e = cudaGetLastError();
    k = q.kout;
    v = q.vout;
  }
  cudaFreeAsync(buf, st);
  return e;
}

cudaError_t radix_run(const RadixPass &io, long long n, const RadixShifts &sh, uint32_t *const t0[2], uint32_t *const t1[2],
                      cudaStream_t st) {
  if (n <= RS_THREADS * RS_FEW) return radix_run_small<RS_FEW>(io, n, sh, st);
  if (n <= RS_THREADS * RS_SMALL) return radix_run_small<RS_SMALL>(io, n, sh, st);
  return n <= RS_FEW_MAX ? radix_run_tiles<RS_FEW>(io, n, sh, t0, t1, st) : radix_run_tiles<RS_ITEMS>(io, n, sh, t0, t1, st);
}

}  // namespace

// Sorts in place (keys / vals) by key bits [0, nbits) using caller scratch of the same size.
cudaError_t radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *ktmp, uint32_t *vtmp, long long n, int nbits,
                             cudaStream_t st) {
  if (n <= 1 || nbits <= 0) return cudaSuccess;
  RadixShifts sh{};
  for (int s = 0; s < nbits && s < 32; s += 8) sh.shift[sh.n++] = s;
  uint32_t *const t[2] = {ktmp, vtmp}, *const o[2] = {keys, vals};
  // through ktmp / vtmp and back; an odd last pass ends there and is copied
  const bool odd = (sh.n & 1) && n > radix_tile(n);
  const RadixPass io{keys, vals, odd ? ktmp : keys, odd ? vtmp : vals, nullptr, 0, 0, 0, 0};
  cudaError_t e = radix_run(io, n, sh, t, o, st);
  if (e == cudaSuccess && odd) e = copy_u32(keys, ktmp, n, st);
  if (e == cudaSuccess && odd) e = copy_u32(vals, vtmp, n, st);
  return e;
}

// `batch` arrays of `len` pairs each, sorted on their own: by key, carrying
// the original index, then by array number.  dir 0 sorts the complements (the
// same order of equal keys).
cudaError_t sort_pairs_batched(uint32_t *dk, uint32_t *dv, const uint32_t *sk, const uint32_t *sv, uint32_t batch,
                               uint32_t len, uint32_t dir, cudaStream_t st) {
  const long long n = (long long)batch * len;
  if (n == 0) return cudaSuccess;
  RadixShifts sh{};
  for (int s = 0; s < 32; s += 8) sh.shift[sh.n++] = s;
  for (int s = 0; batch > 1 && s < 32 && ((batch - 1) >> s) != 0; s += 8) {
    sh.shift[sh.n] = s;
    sh.len[sh.n++] = len;
  }
  const uint32_t x = dir ? 0u : ~0u;
  const RadixPass io{sk, batch > 1 ? nullptr : sv, dk, dv, batch > 1 ? sv : nullptr, x, x, 0, 0};
  uint32_t *buf = nullptr;
  cudaError_t e = cudaSuccess;
  auto meet = [&](const uint32_t *a, const uint32_t *b) { return a < b + n && b < a + n; };
  const bool inplace_values = batch > 1 && (meet(sv, dk) || meet(sv, dv));  // the last pass gathers from sv while it writes
  const size_t words = n > radix_tile(n) ? 4 * (size_t)n : 0, extra = inplace_values ? (size_t)n : 0;
  if (words + extra) e = cudaMallocAsync((void **)&buf, sizeof(uint32_t) * (words + extra), st);
  if (e != cudaSuccess) return e;
  uint32_t *const t0[2] = {buf, buf + n}, *const t1[2] = {buf + 2 * n, buf + 3 * n};
  RadixPass run = io;
  if (inplace_values) {
    e = copy_u32(buf + words, sv, n, st);
    run.gather = buf + words;
  }
  if (e == cudaSuccess) e = radix_run(run, n, sh, t0, t1, st);
  if (buf) cudaFreeAsync(buf, st);
  return e;
}

}  // namespace dmsc
