// grid_kernels.cu -- discrete gradient, critical-cell collation and owner
// labels for one piece of a 2D grid, hand-written for sm_103a.
//
// Restates, as data-parallel tile kernels, the reference CPU path
//   GridDataset::assignGradients        dmsc/src/grid_dataset.cpp:1743-1820
//   lowestPairableCoFacet               dmsc/src/grid_dataset.cpp:1314-1373
//   compareCells / ptLt                 grid_dataset.cpp:1519-1536, grid_dataset.h:158-167
//   GridDataset::collateCriticalPoints  grid_dataset.cpp:1822-1832
//   assignCellOwnerExtrema + BFS        grid_dataset.cpp:1376-1427, 1835-1856
//   writeout_connectivity (arcs, fns)   grid_dataset.cpp:1538-1552, 1858-1907
//
// Vertex order.  ptLt compares values, then cell ids lexicographically; a
// vertex key is (order-preserving value bits << 32 | x << 16 | y), so ptLt is
// a 64-bit integer compare.  compareCells sorts cell vertices ASCENDING and
// compares lexicographically; two closed forms replace the sorts:
//   * two faces sharing an edge differ in two vertices each, and ascending-
//     sorted lexicographic order puts first the face holding the smallest
//     vertex of the symmetric difference;
//   * edge e=(P,Q) is >= every edge of a face whose other corners are U
//     (adjacent to P) and W (adjacent to Q) iff U<Q and W<P (the "usable" test
//     of lowestPairableCoFacet, :1344-1351): the face's two diagonals are
//     compared, so exactly one of its four edges, the one between the larger
//     ends of both diagonals, is usable for it.
// The reference's OpenCL kernels (work_ocl) sort cell vertices DESCENDING
// instead (dmsc/resources/assigngradient.cl:40-87).  A face's largest edge is
// the same there (the face's largest vertex is the larger end of its diagonal
// and its larger neighbour that of the other one); GridGeom::desc selects the
// mirrored rule for the rest:
//   * two faces sharing an edge are ordered by the LARGEST vertex of their
//     symmetric difference: the face holding it is the larger one.
// A vertex pairs with the edge to its lowest lower neighbour in both orders.
// With either order the other steps of work_ocl (complete_pairings, the two
// boundary-pair kernels, pointer-jumping owners, saddle incidences) give the
// cells and owners of the CPU path's steps.
//
// Exactness of the parallel gradient.  The reference pairs cells in row-major
// order and skips cells already marked.  A cell can only be chosen by its
// unique maximal facet, and a vertex v choosing edge e=(w,v) (w its lowest
// usable lower neighbour) makes e fail the usable test for both of its faces
// (the face edge (v,y) beats e), so no cell is both chosen and choosing and
// row-major order never matters: pair(v) = cand(v); pair(e) = its choosing
// vertex, else cand(e); pair(f) = its choosing edge.  ST_PAIR_CONFLICT flags
// the (impossible) mixed case.
//
// Owner labels.  own() of a non-critical vertex is own() of the far end of
// its paired edge; of a non-critical face, own() of the face across its
// paired edge; of a non-critical edge, own() of its pair.  Critical cells own
// themselves; non-critical exterior cells are never reached (LABEL_NONE).
// K1 follows the V-paths by pointer jumping in shared memory inside a tile
// and writes each cell's in-tile terminal; paths leaving the tile end at a
// border cell, and only the border table is resolved globally (K3).
#include <algorithm>

#include "dmsc_common.cuh"
#include "dmsc_internal.h"
#include "smem_limit.h"

namespace dmsc {

__device__ __forceinline__ bool in_rect(const GridGeom &g, int x, int y) {
  return x >= g.rx0 && x <= g.rx1 && y >= g.ry0 && y <= g.ry1;
}
// True if cell (x,y) (relative to ext) has a cofacet inside ext but outside
// rect.  Only meaningful for cells inside rect (isCellExterior, :1708-1711).
__device__ __forceinline__ bool has_ext_cofacet(const GridGeom &g, int x, int y) {
  int kind = (x & 1) | ((y & 1) << 1);
  bool up = (y == g.ry1 && y + 1 <= g.cy), dn = (y == g.ry0 && y >= 1);
  bool lf = (x == g.rx0 && x >= 1), rt = (x == g.rx1 && x + 1 <= g.cx);
  switch (kind) {
    case 0: return up || dn || lf || rt;  // vertex: four edges
    case 1: return up || dn;              // horizontal edge: faces above/below
    case 2: return lf || rt;              // vertical edge: faces left/right
    default: return false;                // face: no cofacets
  }
}
__device__ __forceinline__ int dir_dx(uint32_t d) { return d == DIR_PX ? 1 : (d == DIR_MX ? -1 : 0); }
__device__ __forceinline__ int dir_dy(uint32_t d) { return d == DIR_PY ? 1 : (d == DIR_MY ? -1 : 0); }

// Gradient code of a cell after the pairing (assignGradients steps 2 and 3):
// unmarked rect cells are critical; the boundary rule marks a paired rect
// cell with an exterior cofacet, and its pair, critical as well.
__device__ __forceinline__ uint32_t finish_code(const GridGeom &g, bool piece, int x, int y, uint32_t dir, bool paired) {
  bool inr = in_rect(g, x, y);
  bool crit = inr && !paired;
  if (piece && paired) {
    if (inr && has_ext_cofacet(g, x, y)) crit = true;
    int px = x + dir_dx(dir), py = y + dir_dy(dir);
    if (in_rect(g, px, py) && has_ext_cofacet(g, px, py)) crit = true;
  }
  return (paired ? (CODE_PAIRED | dir) : 0u) | (crit ? CODE_CRIT : 0u);
}

// The smaller of two faces of an edge by their corners off the edge (two of one
// height: the one further left, then the one further down, is the smaller): true
// if the face below / at the left is.
__device__ __forceinline__ bool lower_face_first(bool desc, uint32_t ul, uint32_t ur, uint32_t dl, uint32_t dr) {
  if (desc) {
    const uint32_t u = max(ul, ur), d = max(dl, dr);
    return u > d || (u == d && !(dr >= dl && ur < ul));
  }
  const uint32_t u = min(ul, ur), d = min(dl, dr);
  return d < u || (d == u && !(dr < dl && ur >= ul));
}
__device__ __forceinline__ bool left_face_first(bool desc, uint32_t r, uint32_t ur, uint32_t l, uint32_t ul) {
  return desc ? max(r, ur) >= max(l, ul) : min(l, ul) <= min(r, ur);
}

// pointer-jumping words (uint16): tag in bits 0-1, local cell index in bits
// 2-13 (a pointer is the byte offset of the word it points to), an EXIT's
// direction in bits 14-15
constexpr uint32_t PJ_PTR = 0, PJ_ROOT = 1, PJ_EXIT = 2, PJ_INVALID = 3, PJ_TAG = 3;
__device__ __forceinline__ uint32_t pj_cell(uint32_t w) { return w >> 2 & 0x0FFF; }

// Jumps every pointer of the tile's words (vertex | face << 16) to its terminal;
// v holds the calling thread's own ROWS words, a column's from entry e0 on.  A
// word read while its owner replaces it is a pointer further along the same
// path, so two hops go between barriers; two such rounds go over all words, the
// rest over those that are still pointers.  Returns true if a path failed to
// terminate (a cycle).
template <int ROWS>
__device__ __forceinline__ bool pointer_jump(uint32_t *pj, uint32_t (&v)[ROWS], int e0) {
  static_assert(ROWS <= 16, "one bit of the mask per word");
  const unsigned char *const at = reinterpret_cast<const unsigned char *>(pj);
  auto word = [&](uint32_t w, int face) -> uint32_t { return *reinterpret_cast<const uint16_t *>(at + 2 * face + w); };
  auto two_hops = [&](uint32_t w, int face) -> uint32_t {
    w = word(w, face);
    return (w & PJ_TAG) == PJ_PTR ? word(w, face) : w;
  };
  uint32_t active = 0;
#pragma unroll
  for (int round = 0; round < 2; ++round) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      uint32_t a = v[k] & 0xFFFFu, b = v[k] >> 16;
      if ((a & PJ_TAG) == PJ_PTR) a = two_hops(a, 0);
      if ((b & PJ_TAG) == PJ_PTR) b = two_hops(b, 1);
      v[k] = a | b << 16;
      pj[e0 + k * TX] = v[k];
      if (round == 1)
        active |= ((a & PJ_TAG) == PJ_PTR ? 1u << k : 0u) | ((b & PJ_TAG) == PJ_PTR ? 0x10000u << k : 0u);
    }
  }
  uint16_t *const half = reinterpret_cast<uint16_t *>(pj);
  for (int round = 2; round < 16; ++round) {  // (9 would do: every round multiplies the hops done by 3)
    if (!__syncthreads_or(active != 0)) return false;
    for (uint32_t m = active; m; m &= m - 1) {
      const int k = __ffs(m) - 1, e = 2 * (e0 + (k & 15) * TX) + (k >> 4);
      const uint32_t w = two_hops(half[e], k >> 4);
      half[e] = (uint16_t)w;
      if ((w & PJ_TAG) != PJ_PTR) active &= ~(1u << k);
    }
  }
  const bool bad = __syncthreads_or(active != 0);
  if (bad) {
    for (uint32_t m = active; m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      half[2 * (e0 + (k & 15) * TX) + (k >> 4)] = (uint16_t)PJ_INVALID;
    }
    __syncthreads();
  }
  return bad;
}

// A tile row's critical cells: crit[half] holds a word per cell kind (V, H, Vt,
// F), one bit per vertex of the row's half.  Ranks count the critical cells of
// the cell row (V and H, or Vt and F) before vertex i's.
__device__ __forceinline__ uint32_t crit_before(const uint4 *crit, int i, bool upper) {
  const uint4 m = crit[i >> 5];
  const uint32_t lt = (1u << (i & 31)) - 1u;
  uint32_t r = upper ? __popc(m.z & lt) + __popc(m.w & lt) : __popc(m.x & lt) + __popc(m.y & lt);
  if (i >= 32) r += upper ? __popc(crit[0].z) + __popc(crit[0].w) : __popc(crit[0].x) + __popc(crit[0].y);
  return r;
}
__device__ __forceinline__ uint32_t face_rank(const uint4 *crit, int i) {  // (its Vt comes before it)
  return crit_before(crit, i, true) + ((crit[i >> 5].z >> (i & 31)) & 1u);
}
// the row's masks from a warp's packed codes (32 vertices of one row)
__device__ __forceinline__ uint4 put_crit(uint4 *crit, uint32_t packed, int i) {
  uint4 m = make_uint4(0, 0, 0, 0);
  if (__any_sync(0xffffffffu, packed & 0x08080808u))
    m = make_uint4(__ballot_sync(0xffffffffu, packed & CODE_CRIT), __ballot_sync(0xffffffffu, packed & (CODE_CRIT << 8)),
                   __ballot_sync(0xffffffffu, packed & (CODE_CRIT << 16)), __ballot_sync(0xffffffffu, packed & (CODE_CRIT << 24)));
  if ((i & 31) == 0) crit[i >> 5] = m;
  return m;
}

// ---------------------------------------------------------------------------
// K1: gradient + in-tile tracing + critical counts + border table
// ---------------------------------------------------------------------------
// What bounds it is instructions, not its 12 bytes a vertex: a thread takes a
// column of 8 (or 16) rows, so that a row costs it three loads of heights (the
// 3x3 neighbourhood slides along in registers) and ten comparisons; a choice is
// at once the code bits of the two cells it pairs, so a quad's codes are the OR
// of three words, and the first step of its tracing is a table's entry; critical cells are counted from ballots.  (Heights are
// compared as 32-bit words, the vertices' positions deciding between equal ones
// by the sign of the offset, known beforehand.)  4096x4096 quantised heights:
// 328 us with one item per cell and step, 177 us so; 1000 grids of 64 to 2048 a
// side: 15.0 ms, 8.3 ms.
struct GradSmem {
  union {
    uint32_t key[TY + 3][TX + 3];  // height of vertex (tx0-1+ii, ty0-1+jj)
    uint32_t pj[TY * TX];          // pointer-jumping words, vertex | face << 16
  };
  uint32_t own[TY + 1][TX + 1];    // code bits set by the choices of a quad's vertex and edges
  uint4 crit[TY][2];
  uint32_t step[16][16];           // [the directions that leave the tile][code]: a word less its cell's offset
};

// The cell of border slot b of a tile with clipped extents (W, H), if there is one.
__device__ __forceinline__ bool border_cell(int b, int W, int H, int &i, int &j) {
  if (b < TX) { i = b; j = 0; }
  else if (b < 2 * TX) { i = b - TX; j = H - 1; }
  else if (b < 2 * TX + TY) { i = 0; j = b - 2 * TX; }
  else { i = W - 1; j = b - 2 * TX - TY; }
  return W > 0 && H > 0 && i >= 0 && i < W && j >= 0 && j < H && border_index(i, j, W, H) == b;
}

// True if every cell of tile (bx, by), its one-vertex halo and the cells
// paired across its border lie strictly inside rect and away from the grid's
// border: the bounds tests, the grid-border rule of lowestPairableCoFacet and
// the exterior-cofacet rule then all have fixed outcomes.
__device__ __forceinline__ bool interior_tile(const GridGeom &g, int bx, int by) {
  const int tx0 = bx * TX, ty0 = by * TY;
  return tx0 >= 2 && ty0 >= 2 && tx0 + TX + 2 < g.vnx && ty0 + TY + 2 < g.vny && g.rx0 + 4 <= 2 * tx0 &&
         g.ry0 + 4 <= 2 * ty0 && 2 * (tx0 + TX) + 4 <= g.rx1 && 2 * (ty0 + TY) + 4 <= g.ry1;
}

// the heights around a vertex: d(own) / u(p) a row below / above, l(eft), r(ight)
struct Around {
  uint32_t dc, dr, l, c, r, ul, uc, ur;
};
// A quad's four codes, V | H << 8 | Vt << 16 | F << 24, as far as the choices of
// its own vertex and edges set them.  A choice to the left or downwards pairs a
// cell of another quad: it also sets the bits that from_right and from_above
// shift into that quad's codes.
constexpr uint32_t V_PX = CODE_PAIRED | DIR_PX | (CODE_PAIRED | DIR_MX) << 8, V_MX = CODE_PAIRED | DIR_MX | 1u << 3,
                   V_PY = CODE_PAIRED | DIR_PY | (CODE_PAIRED | DIR_MY) << 16, V_MY = CODE_PAIRED | DIR_MY | 3u << 4,
                   H_PY = (CODE_PAIRED | DIR_PY) << 8 | (CODE_PAIRED | DIR_MY) << 24,
                   H_MY = (CODE_PAIRED | DIR_MY | 3u << 4) << 8,
                   VT_PX = (CODE_PAIRED | DIR_PX) << 16 | (CODE_PAIRED | DIR_MX) << 24,
                   VT_MX = (CODE_PAIRED | DIR_MX | 1u << 3) << 16;
constexpr uint32_t OWN_CODES = 0x07070707, EDGES_PAIRED = CODE_PAIRED << 8 | CODE_PAIRED << 16;
static_assert((1u << 3) << 7 == (CODE_PAIRED | DIR_PX) << 8 && (3u << 4) << 13 == (CODE_PAIRED | DIR_PY) << 16, "the shifts below");
__device__ __forceinline__ uint32_t from_right(uint32_t own) { return own << 7 & 0x04000400; }
__device__ __forceinline__ uint32_t from_above(uint32_t own) { return own << 13 & 0x06060000; }
// Lowest pairable cofacets of vertex (vi, vj), of the edge to its right and of
// the edge above it (only rect cells choose), as the quad's own code bits.
template <bool INTERIOR>
__device__ __forceinline__ uint32_t choose(const GridGeom &g, const Around &q, int vi, int vj, uint32_t &clash) {
  // the diagonals of the face to the upper right: the top left end is the smaller
  // of the one, the top right end the smaller of the other (a tie goes by x)
  const bool a0 = q.uc <= q.r, b0 = q.ur < q.c;
  uint32_t v = 0, h = 0, t = 0;
  if (INTERIOR || (vi < g.vnx && vj < g.vny && in_rect(g, 2 * vi, 2 * vj))) {
    const bool tbv = !INTERIOR && (vi == 0 || vi == g.vnx - 1 || vj == 0 || vj == g.vny - 1);
    const bool okv = !tbv || vi == 0 || vi == g.vnx - 1;  // vertical edges usable
    const bool okh = !tbv || vj == 0 || vj == g.vny - 1;  // horizontal edges usable
    // minimum over the lower neighbours; equal heights order left, below, own, above, right
    uint32_t low = q.c;
    if (okv && (INTERIOR || vj >= 1) && q.dc <= low) { low = q.dc; v = V_MY; }
    if (okh && (INTERIOR || vi >= 1) && q.l <= low) { low = q.l; v = V_MX; }
    if (okv && (INTERIOR || vj + 1 < g.vny) && q.uc < low) { low = q.uc; v = V_PY; }
    if (okh && (INTERIOR || vi + 1 < g.vnx) && q.r < low) { low = q.r; v = V_PX; }
  }
  // H: the bottom edge of the face above, the top edge of the face below
  if (INTERIOR || (vi + 1 < g.vnx && vj < g.vny && in_rect(g, 2 * vi + 1, 2 * vj) && vj != 0 && vj != g.vny - 1)) {
    const bool above = a0 && b0, below = !(q.c <= q.dr) && !(q.r < q.dc);
    h = below && (!above || lower_face_first(g.desc, q.uc, q.ur, q.dc, q.dr)) ? H_MY : above ? H_PY : 0u;
  }
  // Vt: the left edge of the face at the right, the right edge of the face at the left
  if (INTERIOR || (vi < g.vnx && vj + 1 < g.vny && in_rect(g, 2 * vi, 2 * vj + 1) && vi != 0 && vi != g.vnx - 1)) {
    const bool right = !a0 && b0, left = q.ul <= q.c && !(q.uc < q.l);
    t = left && (!right || left_face_first(g.desc, q.r, q.ur, q.l, q.ul)) ? VT_MX : right ? VT_PX : 0u;
  }
  clash |= v & (h | t);
  return v | h | t;
}

// K1 on tile (bx, by) of one grid, THREADS threads per block; INTERIOR:
// the tile satisfies interior_tile (the same results with fewer tests).
template <int THREADS, bool INTERIOR>
__device__ __forceinline__ void gradient_tile_t(const float *__restrict__ hgt, const GridGeom &g, uint32_t *__restrict__ codes,
                                              uint32_t *__restrict__ terms, uint8_t *__restrict__ rowcnt,
                                              uint64_t *__restrict__ table, uint32_t *__restrict__ status, int bx, int by) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem &s = *reinterpret_cast<GradSmem *>(smem_raw);
  constexpr int ROWS = TX * TY / THREADS;
  const int i = threadIdx.x % TX, j0 = threadIdx.x / TX * ROWS, e0 = j0 * TX + i;
  const int tx0 = bx * TX, ty0 = by * TY;
  int w, h, wf, hf;
  tile_extent(g, bx, by, 0, w, h);
  tile_extent(g, bx, by, 1, wf, hf);
  if (INTERIOR) { w = h = wf = hf = TX; }
  const bool piece = !INTERIOR && !(g.rx0 == 0 && g.ry0 == 0 && g.rx1 == g.cx && g.ry1 == g.cy);
  uint32_t st = 0, clash = 0;  // clash: EDGES_PAIRED bits of edges paired twice

  // 1. heights with a 1-vertex halo below/left and 2 above/right: a warp takes
  //    rows, 64 of their vertices; the last three columns go by threads
  auto load = [&](int ii, int jj) -> float {
    const int vi = tx0 - 1 + ii, vj = ty0 - 1 + jj;
    if (!INTERIOR && !(vi >= 0 && vi < g.vnx && vj >= 0 && vj < g.vny)) return 0.0f;
    return __ldg(hgt + (long long)vj * g.pitch + vi);
  };
  auto keep = [&](int ii, int jj, float f) {
    if (f != f) st |= ST_NAN_INPUT;
    s.key[jj][ii] = ord_key(f);
  };
  constexpr int WARPS = THREADS / 32, AT_ONCE = 5;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int b = 0; b < TY + 3; b += AT_ONCE * WARPS) {
    float f[AT_ONCE][2];
#pragma unroll
    for (int q = 0; q < AT_ONCE; ++q) {
      const int jj = b + q * WARPS + warp;
      if (jj < TY + 3) { f[q][0] = load(lane, jj); f[q][1] = load(lane + 32, jj); }
    }
#pragma unroll
    for (int q = 0; q < AT_ONCE; ++q) {
      const int jj = b + q * WARPS + warp;
      if (jj < TY + 3) { keep(lane, jj, f[q][0]); keep(lane + 32, jj, f[q][1]); }
    }
  }
  if (INTERIOR && threadIdx.x < 256) {
    const uint32_t leaves = threadIdx.x >> 4, d = threadIdx.x & 3, by = d & 2 ? 4 * TX : 4;
    (&s.step[0][0])[threadIdx.x] = threadIdx.x & CODE_CRIT ? PJ_ROOT : leaves >> d & 1 ? PJ_EXIT | d << 14 : d & 1 ? 0u - by : by;
  }
  static_assert(3 * (TY + 3) <= THREADS && THREADS >= 256, "the last columns in one go");
  if (threadIdx.x < 3 * (TY + 3)) {
    const int jj = threadIdx.x / 3, ii = TX + threadIdx.x % 3;
    keep(ii, jj, load(ii, jj));
  }
  __syncthreads();

  // 2. lowest pairable cofacets of the tile's vertices and edges, then those of
  //    the column to the right and the row above
  {
    const uint32_t *k = &s.key[j0][i + 1];  // a row below, own column
    Around q;
    q.l = k[-1 + (TX + 3)]; q.c = k[TX + 3]; q.r = k[1 + (TX + 3)];
    q.dc = k[0]; q.dr = k[1];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const uint32_t *u = k + (r + 2) * (TX + 3);
      q.ul = u[-1]; q.uc = u[0]; q.ur = u[1];
      s.own[j0 + r][i] = choose<INTERIOR>(g, q, tx0 + i, ty0 + j0 + r, clash);
      q.dc = q.c; q.dr = q.r;
      q.l = q.ul; q.c = q.uc; q.r = q.ur;
    }
  }
  if (threadIdx.x < TX + TY + 1) {
    const int ii = threadIdx.x <= TY ? TX : threadIdx.x - TY - 1, jj = threadIdx.x <= TY ? threadIdx.x : TY;
    const uint32_t *k = &s.key[jj + 1][ii + 1], *d = k - (TX + 3), *u = k + (TX + 3);
    s.own[jj][ii] = choose<INTERIOR>(g, Around{d[0], d[1], k[-1], k[0], k[1], u[-1], u[0], u[1]}, tx0 + ii, ty0 + jj, clash);
  }
  __syncthreads();  // (the heights are dead from here on: the tracing's words take their place)

  // 3. final codes of the tile's own cells; the first step of the in-tile
  //    tracing: vertices follow their paired edge to the next vertex, faces
  //    follow their paired edge to the face across it
  uint32_t v[ROWS], above = s.own[j0][i];
  const uint32_t sideways = (i == w - 1 ? 1u << DIR_PX : 0u) | (i == 0 ? 1u << DIR_MX : 0u);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int j = j0 + r;
    const uint32_t e = e0 + r * TX, own = above;
    above = s.own[j + 1][i];
    const uint32_t fr = from_right(s.own[j][i + 1]), fa = from_above(above);
    uint32_t packed = (own & OWN_CODES) | fr | fa;
    clash |= (own & (fr | fa)) | (fr & fa);
    const int vi = tx0 + i, vj = ty0 + j, x = 2 * vi, y = 2 * vj;
    if (INTERIOR) {
      packed |= (~packed & 0x04040404u) << 1;  // what is not paired is critical
      const uint32_t leaves = sideways | (r == ROWS - 1 && j == TY - 1 ? 1u << DIR_PY : 0u) | (r == 0 && j == 0 ? 1u << DIR_MY : 0u);
      const uint32_t *const step = s.step[leaves];
      v[r] = (4 * e + step[packed & 15]) | (4 * e + step[packed >> 24]) << 16;
      codes[(long long)vj * g.vnx + vi] = packed;
    } else {
      uint32_t pvv = PJ_INVALID, pff = PJ_INVALID, c = 0;
      if (i < w && j < h) {
#pragma unroll
        for (int kind = 0; kind < 4; ++kind)
          if (((kind & 1) == 0 || vi + 1 < g.vnx) && ((kind & 2) == 0 || vj + 1 < g.vny))
            c |= finish_code(g, piece, x + (kind & 1), y + (kind >> 1), packed >> (8 * kind) & 3, packed >> (8 * kind) & CODE_PAIRED)
                 << (8 * kind);
        codes[(long long)vj * g.vnx + vi] = c;
        auto step = [&](uint32_t code, int ww, int hh) -> uint32_t {
          const uint32_t d = code & 3;
          const int ni = i + dir_dx(d), nj = j + dir_dy(d);
          return ni >= 0 && ni < ww && nj >= 0 && nj < hh ? PJ_PTR | (uint32_t)(nj * TX + ni) << 2 : PJ_EXIT | d << 14 | e << 2;
        };
        if (c & CODE_CRIT) pvv = PJ_ROOT | e << 2;
        else if (in_rect(g, x, y)) pvv = step(c, w, h);
        if (i < wf && j < hf) {
          if (c & (CODE_CRIT << 24)) pff = PJ_ROOT | e << 2;
          else if (in_rect(g, x + 1, y + 1)) pff = step(c >> 24, wf, hf);
        }
      }
      packed = c;
      v[r] = pvv | pff << 16;
    }
    s.pj[e] = v[r];
    put_crit(s.crit[j], packed, i);
  }
  if (clash & EDGES_PAIRED) st |= ST_PAIR_CONFLICT;
  if (pointer_jump<ROWS>(s.pj, v, e0)) st |= ST_CYCLE;  // (begins with a barrier)

  // 4. in-tile terminals of every vertex and face, per (cell row, tile) counts
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
    if (i < w && j0 + r < h)
      terms[(long long)(ty0 + j0 + r) * g.vnx + tx0 + i] = s.pj[e0 + r * TX];
  for (int j = threadIdx.x; j < h; j += blockDim.x) {
    const int y = 2 * (ty0 + j);
    const uint4 a = s.crit[j][0], b = s.crit[j][1];
    rowcnt[(long long)y * g.ntx + bx] = (uint8_t)(__popc(a.x) + __popc(a.y) + __popc(b.x) + __popc(b.y));
    if (y + 1 <= g.cy) rowcnt[(long long)(y + 1) * g.ntx + bx] = (uint8_t)(__popc(a.z) + __popc(a.w) + __popc(b.z) + __popc(b.w));
  }

  // 5. border table: where each border cell's path ends inside this tile
  long long tile_base = ((long long)by * g.ntx + bx) * SLOTS_PER_TILE;
  for (int e = threadIdx.x; e < 2 * SLOTS_SIDE; e += blockDim.x) {
    int kind = e / SLOTS_SIDE, b = e - kind * SLOTS_SIDE;
    int W = kind ? wf : w, H = kind ? hf : h;
    int bi, bj;
    const bool there = border_cell(b, W, H, bi, bj);
    uint64_t entry = BT_INVALID;
    if (there) {
      const uint16_t p = (uint16_t)(s.pj[bj * TX + bi] >> (16 * kind));
      const int k = pj_cell(p), ki = k % TX, kj = k / TX;
      if ((p & PJ_TAG) == PJ_ROOT) {
        const int y = 2 * (ty0 + kj) + kind;
        const uint32_t rank = kind ? face_rank(s.crit[kj], ki) : crit_before(s.crit[kj], ki, false);
        entry = BT_ROOT | ((uint64_t)((long long)y * g.ntx + bx + g.gbase) << 8) | rank;
      } else if ((p & PJ_TAG) == PJ_EXIT) {
        const uint32_t d = p >> 14;
        const int gi = tx0 + ki + dir_dx(d), gj = ty0 + kj + dir_dy(d);
        if (gi >= 0 && gj >= 0 && gi < g.vnx - kind && gj < g.vny - kind) entry = BT_EXIT | (uint64_t)(border_slot(g, kind, gi, gj) + g.sbase);
        else st |= ST_CYCLE;  // a path leaving the window: never expected
      }
    }
    table[tile_base + kind * SLOTS_SIDE + b] = entry;
  }
  if (st) atomicOr(status, st);
}
template <int THREADS>
__device__ __forceinline__ void gradient_tile(const float *__restrict__ hgt, const GridGeom &g, uint32_t *__restrict__ codes,
                                              uint32_t *__restrict__ terms, uint8_t *__restrict__ rowcnt,
                                              uint64_t *__restrict__ table, uint32_t *__restrict__ status, int bx, int by) {
  if (interior_tile(g, bx, by))
    gradient_tile_t<THREADS, true>(hgt, g, codes, terms, rowcnt, table, status, bx, by);
  else
    gradient_tile_t<THREADS, false>(hgt, g, codes, terms, rowcnt, table, status, bx, by);
}

__global__ void __launch_bounds__(GRAD_THREADS, 3)
k_gradient(const float *__restrict__ hgt, GridGeom g, uint32_t *__restrict__ codes, uint32_t *__restrict__ terms,
           uint8_t *__restrict__ rowcnt, uint64_t *__restrict__ table, uint32_t *__restrict__ status) {
  gradient_tile<GRAD_THREADS>(hgt, g, codes, terms, rowcnt, table, status, blockIdx.x, blockIdx.y);
}

// The grid of batch tile t (tiles numbered grid after grid).
__device__ __forceinline__ int batch_grid_of(const BatchGrid *G, int ngrids, long long t) {
  int lo = 0, hi = ngrids - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (G[mid].tile0 <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// K1 over a batch: a persistent grid of blocks takes (grid, tile) items in
// order; THREADS threads per block (the launch configurations of the batch's
// autotuner).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 3)
k_gradient_batch(const BatchGrid *__restrict__ G, int ngrids, long long ntiles, uint32_t *__restrict__ status) {
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchGrid B = G[batch_grid_of(G, ngrids, t)];  // (a copy: the tile's stores cannot change it)
    const int lt = (int)(t - B.tile0);
    gradient_tile<THREADS>(B.hgt, B.g, B.codes, B.terms, B.rowcnt, B.table, status, lt % B.g.ntx, lt / B.g.ntx);
    __syncthreads();  // shared memory is reused by the next item
  }
}

// ---------------------------------------------------------------------------
// K3: resolve the border table.  Every EXIT chain is followed to its root;
// pointers are compressed in place (any value a reader sees is a valid
// pointer along the same chain), so no grid-wide barrier is needed.
// ---------------------------------------------------------------------------
__global__ void k_resolve(uint64_t *table, long long nslots, const uint32_t *__restrict__ offsets, long long nseg,
                          uint32_t *__restrict__ status) {
  for (long long sidx = blockIdx.x * (long long)blockDim.x + threadIdx.x; sidx < nslots;
       sidx += (long long)gridDim.x * blockDim.x) {
    volatile uint64_t *vt = table;
    uint64_t e = vt[sidx];
    long long iter = 0;
    while (bt_tag(e) == BT_EXIT) {
      if ((long long)bt_payload(e) >= nslots) { e = BT_INVALID; atomicOr(status, ST_RESOLVE_LIMIT); break; }
      uint64_t t = vt[bt_payload(e)];
      e = t;
      if (bt_tag(e) == BT_EXIT) vt[sidx] = e;
      if (++iter > nslots) { e = BT_INVALID; atomicOr(status, ST_RESOLVE_LIMIT); break; }
    }
    if (bt_tag(e) == BT_ROOT) {
      uint64_t pl = bt_payload(e);
      if ((long long)(pl >> 8) < nseg) e = BT_FINAL | (uint64_t)(offsets[pl >> 8] + (uint32_t)(pl & 0xff));
      else { e = BT_INVALID; atomicOr(status, ST_RESOLVE_LIMIT); }
    }
    vt[sidx] = e;
  }
}

// ---------------------------------------------------------------------------
// K4: owner labels, critical-point records and saddle arcs.
// ---------------------------------------------------------------------------
struct LabelSmem {
  // labels of the tile's vertices, and of those one past it to the right and
  // above; of its faces, and of those one before it to the left and below
  uint32_t labV[TY + 1][TX + 1], labF[TY + 1][TX + 1];
  uint4 crit[TY][2];
  uint32_t offA[TY], offB[TY];
  uint32_t nsaddle, nextremum;
  uint16_t list[4 * TY * TX];  // critical cells, (cell << 2 | kind): saddles from the front, extrema from the back
};

__device__ __forceinline__ uint32_t final_label(uint64_t e) { return bt_tag(e) == BT_FINAL ? (uint32_t)bt_payload(e) : LABEL_NONE; }
__device__ __forceinline__ uint32_t slot_label(const uint64_t *table, const GridGeom &g, int kind, int gi, int gj) {
  return final_label(table[border_slot(g, kind, gi, gj)]);
}
__device__ __forceinline__ float hat(const float *hgt, const GridGeom &g, int vi, int vj) {
  return __ldg(hgt + (long long)vj * g.pitch + vi);
}
// get_cell_fn (:1538-1552): float sum in getCellPoints order, then / count.
__device__ __forceinline__ float cell_fn(const float *hgt, const GridGeom &g, int kind, int vi, int vj) {
  float fn = 0.0f;
  switch (kind) {
    case 0: fn = __fadd_rn(fn, hat(hgt, g, vi, vj)); return __fdiv_rn(fn, 1.0f);
    case 1: fn = __fadd_rn(fn, hat(hgt, g, vi + 1, vj)); fn = __fadd_rn(fn, hat(hgt, g, vi, vj)); return __fdiv_rn(fn, 2.0f);
    case 2: fn = __fadd_rn(fn, hat(hgt, g, vi, vj + 1)); fn = __fadd_rn(fn, hat(hgt, g, vi, vj)); return __fdiv_rn(fn, 2.0f);
    default:
      fn = __fadd_rn(fn, hat(hgt, g, vi + 1, vj + 1));
      fn = __fadd_rn(fn, hat(hgt, g, vi + 1, vj));
      fn = __fadd_rn(fn, hat(hgt, g, vi, vj));
      fn = __fadd_rn(fn, hat(hgt, g, vi, vj + 1));
      return __fdiv_rn(fn, 4.0f);
  }
}

// K4 on tile (bx, by) of one grid, THREADS threads per block; INTERIOR: the
// tile satisfies interior_tile.  Its 24 bytes a vertex take less time than its
// instructions: each thread keeps the codes of its column's rows in registers;
// the labels of border cells, in the tile and around it, are read from the
// border table once; critical cells find their index from the rows' ballots; and
// where those leave them every other cell's terminal finds its label.  Records
// go by a list of the tile's critical cells, so that no lane waits for another's.
// 4096x4096 quantised heights: 276 us with a look into the table for every path
// that leaves the tile and records by their cells' threads, 161 us so; 1000 grids
// of 64 to 2048 a side: 9.1 ms, 6.5 ms.
template <int THREADS, bool INTERIOR>
__device__ __forceinline__ void labels_tile_t(const uint32_t *__restrict__ codes, const uint32_t *__restrict__ terms,
                                              const float *__restrict__ hgt, const GridGeom &g,
                                              const uint32_t *__restrict__ offsets, const uint64_t *__restrict__ table,
                                              uint4 *__restrict__ labels, const CpOut &cp, uint32_t *__restrict__ status,
                                              int bx, int by) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LabelSmem &s = *reinterpret_cast<LabelSmem *>(smem_raw);
  constexpr int ROWS = TX * TY / THREADS;
  const int i = threadIdx.x % TX, j0 = threadIdx.x / TX * ROWS, e0 = j0 * (TX + 1) + i;
  const int tx0 = bx * TX, ty0 = by * TY;
  int w, h, wf, hf;
  tile_extent(g, bx, by, 0, w, h);
  tile_extent(g, bx, by, 1, wf, hf);
  if (INTERIOR) { w = h = wf = hf = TX; }
  uint32_t st = 0;
  uint32_t *const labV = &s.labV[0][0], *const labF = &s.labF[1][1];  // entry (i, j) at j * LS + i
  constexpr int LS = TX + 1;

  // arrays too small for the critical points: nothing is done (the caller grows
  // them and calls again; 4096x4096 quantised heights: 0.15 ms of labels saved)
  if (cp.count && *cp.count > cp.cap) {
    if (threadIdx.x == 0) atomicOr(status, ST_CAPACITY);
    return;
  }
  uint32_t code[ROWS], term[ROWS];
  const long long at0 = (long long)(ty0 + j0) * g.vnx + tx0 + i;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    code[r] = 0;
    term[r] = PJ_INVALID | (uint32_t)PJ_INVALID << 16;
    if (i < w && j0 + r < h) {
      code[r] = codes[at0 + (long long)r * g.vnx];
      term[r] = terms[at0 + (long long)r * g.vnx];
    }
  }
  for (int j = threadIdx.x; j < h; j += blockDim.x) {
    int y = 2 * (ty0 + j);
    s.offA[j] = offsets[(long long)y * g.ntx + bx];
    s.offB[j] = (y + 1 <= g.cy) ? offsets[(long long)(y + 1) * g.ntx + bx] : 0u;
  }
  // the border table's labels: border cells, then the cells around the tile
  for (int q = threadIdx.x; q < 2 * SLOTS_SIDE; q += THREADS) {
    const int kind = q / SLOTS_SIDE, b = q - kind * SLOTS_SIDE;
    int bi, bj;
    if (border_cell(b, kind ? wf : w, kind ? hf : h, bi, bj))
      (kind ? labF : labV)[bj * LS + bi] = final_label(table[((long long)by * g.ntx + bx) * SLOTS_PER_TILE + q]);
  }
  for (int q = threadIdx.x; q < 2 * (TX + TY); q += THREADS) {
    const int n = q & (TX - 1), kind = q / (TX + TY);
    const bool row = q & TX;
    const int ii = row ? n : kind ? -1 : TX, jj = row ? (kind ? -1 : TY) : n;
    const int gi = tx0 + ii, gj = ty0 + jj;
    (kind ? labF : labV)[jj * LS + ii] =
        gi >= 0 && gj >= 0 && gi < g.vnx - kind && gj < g.vny - kind ? slot_label(table, g, kind, gi, gj) : LABEL_NONE;
  }
  if (threadIdx.x == 0) s.nsaddle = s.nextremum = 0;
  __syncthreads();
  {  // the tile's critical cells, in no order: each warp takes room for its rows'
    uint32_t ns = 0, ne = 0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const uint4 m = put_crit(s.crit[j0 + r], code[r], i);
      ns += __popc(m.y) + __popc(m.z);
      ne += __popc(m.x) + __popc(m.w);
    }
    uint32_t ps = 0, pe = 0;
    if ((i & 31) == 0) {
      if (ns) ps = atomicAdd(&s.nsaddle, ns);
      if (ne) pe = atomicAdd(&s.nextremum, ne);
    }
    ps = __shfl_sync(0xffffffffu, ps, 0);
    pe = 4 * TY * TX - 1 - __shfl_sync(0xffffffffu, pe, 0);
    const uint32_t lt = (1u << (i & 31)) - 1u;
    if (ns + ne) {
#pragma unroll 1
      for (int r = 0; r < ROWS; ++r) {
        const uint4 m = s.crit[j0 + r][i >> 5];
        const uint32_t e = (uint32_t)((j0 + r) * TX + i) << 2;
        if (m.x >> (i & 31) & 1) s.list[pe - __popc(m.x & lt)] = (uint16_t)e;
        pe -= __popc(m.x);
        if (m.w >> (i & 31) & 1) s.list[pe - __popc(m.w & lt)] = (uint16_t)(e | 3);
        pe -= __popc(m.w);
        if (m.y >> (i & 31) & 1) s.list[ps + __popc(m.y & lt)] = (uint16_t)(e | 1);
        ps += __popc(m.y);
        if (m.z >> (i & 31) & 1) s.list[ps + __popc(m.z & lt)] = (uint16_t)(e | 2);
        ps += __popc(m.z);
      }
    }
  }
  __syncthreads();

  // critical vertices and faces: their own indices
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int j = j0 + r;
    if (code[r] & CODE_CRIT) labV[e0 + r * LS] = s.offA[j] + crit_before(s.crit[j], i, false);
    if (code[r] & (CODE_CRIT << 24)) labF[e0 + r * LS] = s.offB[j] + face_rank(s.crit[j], i);
  }
  __syncthreads();
  // the others: the labels where their paths end (only critical and border
  // cells' entries are read here, and only the others' are written)
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int j = j0 + r;
    auto end = [&](uint32_t p, const uint32_t *lab) -> uint32_t {
      const uint32_t k = pj_cell(p);
      return (p & PJ_TAG) == PJ_ROOT || (p & PJ_TAG) == PJ_EXIT ? lab[k + k / TX] : LABEL_NONE;
    };
    if (!(code[r] & CODE_CRIT) && !on_tile_border(i, j, w, h)) labV[e0 + r * LS] = end(term[r] & 0xffff, labV);
    if (!(code[r] & (CODE_CRIT << 24)) && !(i < wf && j < hf && on_tile_border(i, j, wf, hf)))
      labF[e0 + r * LS] = end(term[r] >> 16, labF);
  }
  __syncthreads();

#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int j = j0 + r, e = e0 + r * LS;
    if (i >= w || j >= h) continue;
    const int vi = tx0 + i, vj = ty0 + j, x = 2 * vi, y = 2 * vj;
    const uint32_t c = code[r];
    // a paired edge has the label of the cell it is paired with
    uint32_t L[4];
    L[0] = labV[e];
    L[3] = labF[e];
    L[1] = LABEL_NONE;  // H(i,j)
    if (c & (CODE_CRIT << 8)) L[1] = s.offA[j] + crit_before(s.crit[j], i, false) + (c >> 3 & 1);
    const uint32_t ch = c >> 8, dh = ch & 3;
    if ((ch & (CODE_PAIRED | CODE_CRIT)) == CODE_PAIRED && (INTERIOR || (vi + 1 < g.vnx && in_rect(g, x + 1, y)))) {
      L[1] = dh & 2 ? labF[e - (dh & 1 ? LS : 0)] : labV[e + (dh & 1 ? 0 : 1)];
    }
    L[2] = LABEL_NONE;  // Vt(i,j)
    if (c & (CODE_CRIT << 16)) L[2] = s.offB[j] + crit_before(s.crit[j], i, true);
    const uint32_t ct = c >> 16, dt = ct & 3;
    if ((ct & (CODE_PAIRED | CODE_CRIT)) == CODE_PAIRED && (INTERIOR || (vj + 1 < g.vny && in_rect(g, x, y + 1)))) {
      L[2] = dt & 2 ? labV[e + (dt & 1 ? 0 : LS)] : labF[e - (dt & 1)];
    }
    labels[(long long)vj * g.vnx + vi] = make_uint4(L[0], L[1], L[2], L[3]);
  }

  // critical-point records
  auto record = [&](uint32_t k, int kind, int ci, int cj) -> bool {  // false: no room
    if ((long long)k >= cp.cap) { st |= ST_CAPACITY; return false; }
    const int vi = tx0 + ci, vj = ty0 + cj, cxr = 2 * vi + (kind & 1), cyr = 2 * vj + (kind >> 1);
    const uint32_t cc = codes[(long long)vj * g.vnx + vi] >> (8 * kind) & 0xff;
    cp.cellid[k] = pack_cellid(g.ex0 + cxr, g.ey0 + cyr);
    cp.fn[k] = cell_fn(hgt, g, kind, vi, vj);
    cp.flags[k] = (cc & CODE_PAIRED) ? 1 : 0;
    if (cc & CODE_PAIRED) {
      const uint32_t d = cc & 3;
      cp.pair_cell[k] = pack_cellid(g.ex0 + cxr + dir_dx(d), g.ey0 + cyr + dir_dy(d));
    }
    return true;
  };
  const uint32_t ns = s.nsaddle, ne = s.nextremum;
  for (uint32_t q = threadIdx.x; q < ns; q += THREADS) {
    const uint32_t u = s.list[q], e = u >> 2, kind = u & 3;
    const int ci = e % TX, cj = e / TX, vi = tx0 + ci, vj = ty0 + cj;
    const uint32_t k = kind == 1 ? s.offA[cj] + crit_before(s.crit[cj], ci, false) + (s.crit[cj][ci >> 5].x >> (ci & 31) & 1)
                                 : s.offB[cj] + crit_before(s.crit[cj], ci, true);
    if (!record(k, kind, ci, cj)) continue;
    // facets f[0..1] and ext-filtered cofacets (writeout_connectivity, :1876-1898)
    const uint32_t le = e + cj, f1 = labV[le], f0 = labV[le + (kind == 1 ? 1 : LS)];
    const bool after = kind == 1 ? vj + 1 < g.vny : vi + 1 < g.vnx, before = kind == 1 ? vj >= 1 : vi >= 1;
    const uint32_t q0 = after ? labF[le] : LABEL_NONE, q1 = before ? labF[(int)le - (kind == 1 ? LS : 1)] : LABEL_NONE;
    const uint32_t dlo = min(f0, f1), dhi = max(f0, f1), alo = min(q0, q1), ahi = max(q0, q1);
    cp.des2[2 * k] = dlo; cp.des2[2 * k + 1] = dhi;
    cp.asc2[2 * k] = alo; cp.asc2[2 * k + 1] = ahi;
    cp.dcnt[k] = (dlo != LABEL_NONE) + (dhi != LABEL_NONE);
    cp.acnt[k] = (alo != LABEL_NONE) + (ahi != LABEL_NONE);
    if (dlo != LABEL_NONE && dlo < cp.cap) atomicAdd(cp.acnt + dlo, 1u);
    if (dhi != LABEL_NONE && dhi < cp.cap) atomicAdd(cp.acnt + dhi, 1u);
    if (alo != LABEL_NONE && alo < cp.cap) atomicAdd(cp.dcnt + alo, 1u);
    if (ahi != LABEL_NONE && ahi < cp.cap) atomicAdd(cp.dcnt + ahi, 1u);
  }
  for (uint32_t q = threadIdx.x; q < ne; q += THREADS) {
    const uint32_t u = s.list[4 * TY * TX - 1 - q], e = u >> 2, kind = u & 3;
    const uint32_t k = (kind ? labF : labV)[e + e / TX];
    if (!record(k, kind, e % TX, e / TX)) continue;
    cp.des2[2 * k] = cp.des2[2 * k + 1] = LABEL_NONE;
    cp.asc2[2 * k] = cp.asc2[2 * k + 1] = LABEL_NONE;
  }
  if (st) atomicOr(status, st);
}

template <int THREADS>
__device__ __forceinline__ void labels_tile(const uint32_t *__restrict__ codes, const uint32_t *__restrict__ terms,
                                            const float *__restrict__ hgt, const GridGeom &g,
                                            const uint32_t *__restrict__ offsets, const uint64_t *__restrict__ table,
                                            uint4 *__restrict__ labels, const CpOut &cp, uint32_t *__restrict__ status,
                                            int bx, int by) {
  if (interior_tile(g, bx, by))
    labels_tile_t<THREADS, true>(codes, terms, hgt, g, offsets, table, labels, cp, status, bx, by);
  else
    labels_tile_t<THREADS, false>(codes, terms, hgt, g, offsets, table, labels, cp, status, bx, by);
}

__global__ void __launch_bounds__(GRAD_THREADS, 3)
k_labels(const uint32_t *__restrict__ codes, const uint32_t *__restrict__ terms, const float *__restrict__ hgt, GridGeom g,
         const uint32_t *__restrict__ offsets, const uint64_t *__restrict__ table, uint4 *__restrict__ labels,
         CpOut cp, uint32_t *__restrict__ status) {
  labels_tile<GRAD_THREADS>(codes, terms, hgt, g, offsets, table, labels, cp, status, blockIdx.x, blockIdx.y);
}

// K4 over a batch; cp indices (and so labels) are batch-wide.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 3)
k_labels_batch(const BatchGrid *__restrict__ G, int ngrids, long long ntiles, CpOut cp, uint32_t *__restrict__ status) {
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchGrid B = G[batch_grid_of(G, ngrids, t)];
    const int lt = (int)(t - B.tile0);
    labels_tile<THREADS>(B.codes, B.terms, B.hgt, B.g, B.offsets, B.table, B.labels, cp, status, lt % B.g.ntx, lt / B.g.ntx);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
size_t grad_smem_bytes() { return sizeof(GradSmem); }
size_t label_smem_bytes() { return sizeof(LabelSmem); }

cudaError_t launch_gradient(const float *hgt, const GridGeom &g, uint32_t *codes, uint32_t *terms, uint8_t *rowcnt,
                            uint64_t *table, uint32_t *status, cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = limit.raise(sizeof(GradSmem), k_gradient);
  if (e != cudaSuccess) return e;
  dim3 grid(g.ntx, g.nty);
  k_gradient<<<grid, GRAD_THREADS, sizeof(GradSmem), st>>>(hgt, g, codes, terms, rowcnt, table, status);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

cudaError_t launch_resolve(uint64_t *table, long long nslots, const uint32_t *offsets, long long nseg, uint32_t *status,
                           cudaStream_t st) {
  int threads = 256;
  long long blocks = (nslots + threads - 1) / threads;
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (blocks < 1) blocks = 1;
  k_resolve<<<(unsigned)blocks, threads, 0, st>>>(table, nslots, offsets, nseg, status);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

cudaError_t launch_labels(const uint32_t *codes, const uint32_t *terms, const float *hgt, const GridGeom &g,
                          const uint32_t *offsets, const uint64_t *table, uint4 *labels, const CpOut &cp,
                          uint32_t *status, cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = limit.raise(sizeof(LabelSmem), k_labels);
  if (e != cudaSuccess) return e;
  dim3 grid(g.ntx, g.nty);
  k_labels<<<grid, GRAD_THREADS, sizeof(LabelSmem), st>>>(codes, terms, hgt, g, offsets, table, labels, cp, status);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

// The persistent batch kernels' launch: `threads` per block (256 or 512) and
// blocks_per_sm resident blocks per SM (1 to 3; the shared memory of a 64x64
// tile allows 3) over the device's SMs.
static long long persistent_blocks(long long ntiles, int blocks_per_sm) {
  static const int sms = [] {
    int dev = 0, n = 152;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      n = 152;
    return n;
  }();
  const int bps = blocks_per_sm < 1 ? 1 : blocks_per_sm > 3 ? 3 : blocks_per_sm;
  return std::min<long long>(ntiles, (long long)sms * bps);
}

template <int THREADS>
static cudaError_t gradient_batch_t(const BatchGrid *grids, int ngrids, long long ntiles, int bps, uint32_t *status,
                                    cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = limit.raise(sizeof(GradSmem), k_gradient_batch<THREADS>);
  if (e != cudaSuccess) return e;
  k_gradient_batch<THREADS><<<(unsigned)persistent_blocks(ntiles, bps), THREADS, sizeof(GradSmem), st>>>(grids, ngrids,
                                                                                                      ntiles, status);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

template <int THREADS>
static cudaError_t labels_batch_t(const BatchGrid *grids, int ngrids, long long ntiles, const CpOut &cp, int bps,
                                  uint32_t *status, cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = limit.raise(sizeof(LabelSmem), k_labels_batch<THREADS>);
  if (e != cudaSuccess) return e;
  k_labels_batch<THREADS><<<(unsigned)persistent_blocks(ntiles, bps), THREADS, sizeof(LabelSmem), st>>>(grids, ngrids,
                                                                                                     ntiles, cp, status);
  DMSC_LAUNCHED(1);
  return cudaGetLastError();
}

cudaError_t launch_gradient_batch(const BatchGrid *grids, int ngrids, long long ntiles, uint32_t *status, cudaStream_t st,
                                  BatchLaunch cfg) {
  if (ntiles <= 0) return cudaSuccess;
  return cfg.threads == 256 ? gradient_batch_t<256>(grids, ngrids, ntiles, cfg.blocks_per_sm, status, st)
                            : gradient_batch_t<GRAD_THREADS>(grids, ngrids, ntiles, cfg.blocks_per_sm, status, st);
}

cudaError_t launch_labels_batch(const BatchGrid *grids, int ngrids, long long ntiles, const CpOut &cp, uint32_t *status,
                                cudaStream_t st, BatchLaunch cfg) {
  if (ntiles <= 0) return cudaSuccess;
  return cfg.threads == 256 ? labels_batch_t<256>(grids, ngrids, ntiles, cp, cfg.blocks_per_sm, status, st)
                            : labels_batch_t<GRAD_THREADS>(grids, ngrids, ntiles, cp, cfg.blocks_per_sm, status, st);
}

}  // namespace dmsc
