// Radius search and the matrix-free sparse operator on the GPU.
//
// Reference path restated: KernelSparse::evaluate (src/Kernels.h:720-751)
// calls euclidean_search (src/Search.h:839-845) per row, which walks periodic
// images x buckets of the CellListOrdered grid and accepts a candidate iff
// !(((0+dx0^2)+dx1^2)+dx2^2 > r^2) in FP64 with dx = x_j - (x_i + image*L)
// (src/Search.h:438-465, src/detail/Distance.h:132-137); it then accumulates
// c_i += f(dx, a_i, b_j) * b_j.
//
// GB300 design (not a translation of the bucket-walk iterator):
//  * An internal fine grid of side ~r/3 (padded to 3 dims, last real
//    dimension fastest) re-sorts the column particles so that each (e0,e1)
//    row of fine cells is one contiguous index range; a query tile then
//    visits ~49 contiguous ranges instead of iterating buckets.
//  * Work unit = one warp = up to 32 spatially adjacent queries.  The warp
//    stages 32 candidates at a time in shared memory (one coalesced 16 B load
//    per lane) and every lane tests its query against all of them
//    (broadcast LDS), so each candidate costs one LDS + the pair arithmetic.
//  * Mixed mode: candidate and query coordinates are FP32 offsets from the
//    tile's reference cell (magnitude <= a few cells, so ~1e-9 absolute
//    error).  A pair is accepted outright if d2 <= r2_lo, rejected if
//    d2 > r2_hi, and only inside that rounding band is the reference's exact
//    FP64 test evaluated, so neighbour decisions are identical to the FP64
//    test.  Kernel values are FP32; each lane sums at most 64 terms in FP32 (32 in
//    either half of a packed sum) before it adds them into an FP64 accumulator.
//  * FP64 mode: neighbours by the same two tests; an accepted pair's kernel value
//    comes from the integer units to FP64 accuracy (fix64.cuh), or by the FP64
//    formula where its parameter or distance is outside what those cover.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "fix64.cuh"
#include "handles.cuh"
#include "unit_work.cuh"

namespace abx {

struct alignas(32) D4 {
  double x, y, z, w;
};

struct FineGrid {
  int dim, eoff;
  int m[3];
  double h[3], inv[3];
  float hf[3];
  double lo[3];
  double L[3];
  int periodic[3];
  int K[3];
  uint32_t ncells;
};

// A point set ordered by fine cell.
struct PointLayout {
  int64_t n = 0;
  DevBuf<uint32_t> perm;  // kernel order -> source index
  DevBuf<int4> cell;      // unclamped fine cell (internal dims)
  DevBuf<float4> loc;     // FP32 offset from the clamped cell corner; .w = clamped c2 bits
  DevBuf<D4> posk;        // FP64 position in kernel order (internal dims, pad = 0)
  DevBuf<uint32_t> keys;  // sorted clamped cell keys
  // fixed-point positions in kernel order (fix64.cuh), where the operator's
  // FP64 product runs on the integer units
  DevBuf<longlong2> fxy;
  DevBuf<long long> fz;
  DevBuf<uint32_t> tmp;   // sort scratch
  void release() {
    perm.release(), cell.release(), loc.release(), posk.release();
    keys.release(), fxy.release(), fz.release(), tmp.release();
  }
};

// Which units' queries k_pairs_thread walks instead of a unit kernel: units of
// fewer than `queries` queries whose own row of the stencil holds at most `row`
// columns (a unit of few queries beside a dense cluster still has a long
// candidate list, which a warp stages faster than a lane walks it) and, where
// `around` is not 0, no row of the whole stencil holds more than that; and none
// at all where they are less than 1 / `fold` of the set (the second launch).
struct Split {
  int queries, row, fold, around;
  bool operator==(const Split &o) const {
    return queries == o.queries && row == o.row && fold == o.fold && around == o.around;
  }
};
// FP64: a unit kernel's lanes idle at ~100 instructions a pair.  N = 100,000 x 50
// with units below 4, 7, 12 queries split: 423, 315, 246 us.  Counts: 698, 669,
// 658 us, but 25.2, 25.4, 25.6 ms for the clustered 4M set.  Mixed products: the
// pair itself is ~10 instructions, so that a unit pays at four queries already
// (4M: 20.6, 20.9, 21.5 ms for the same three); sets of fewer than MIXED_MIN
// rows keep to it altogether (2,000: 13 against 21 us; 12,000: 24 against 31;
// 100,000 x 10: 118 against 78).
// FP64 values outside make_unit's rules cost the unit kernel less (its lanes share
// the FP64 pipe), a lane's long walk as much: only where no walk is long.  30,000
// points in 16 clusters, constant kernel: 285 us without the split, 405 with
// SPLIT_FP64's, 300 to 320 with this; 300,000 uniform 515, 195, 195.  In 1-D a stencil is one
// row, which lanes cannot share: no split (3,000 points, constant 46 -> 31 us).
constexpr Split SPLIT_FP64{12, 1 << 30, 16, 0}, SPLIT_VALUES{12, 1 << 30, 16, 48},
    SPLIT_COUNT{7, 12, 4, 0}, SPLIT_MIXED{4, 6, 3, 0}, SPLIT_NONE{0, 0, 1, 0};
constexpr int64_t MIXED_MIN = 50000;

struct PairLayout {
  FineGrid fg;
  double r = 0;
  uint64_t cols_version = 0, rows_version = 0;
  bool self = true;
  PointLayout cols;
  PointLayout rows_own;
  PointLayout *rows = nullptr;
  DevBuf<uint32_t> cell_start;  // fg.ncells + 1
  // Query units (first query in kernel order, count <= 32): full ones from the
  // front of the array, small ones (Split) from its back, and the latter's
  // queries once more as a list (k_units).
  DevBuf<int2> units;
  DevBuf<int> singles;
  DevBuf<uint8_t> exits;  // of the units' chunks, and their entries (k_unit_exits)
  Split split = SPLIT_NONE;
  // full units, small units, their queries, stencil rows; work counters of a
  // count or product (4, 5) and of a list search (6, 7); small units and single
  // queries that a count or product works (8, 9)
  DevBuf<int> counts;
  // written by k_tables into pinned host memory: one of the two pair kernels has
  // no work at uniform density, and is not launched then (unit_work.cuh)
  uint64_t *work = nullptr;
  uint32_t work_seq = 0;
  ~PairLayout() {
    if (work) cudaFreeHost(work);
  }
  DevBuf<float> bk32;
  DevBuf<double> bk64;
  DevBuf<double> sk;  // column scalar in kernel order
  DevBuf<double> sq;  // row scalar in kernel order
  DevBuf<int> ext;        // e2 extent table
  DevBuf<float4> bands;   // rounding bands by tile span (k_tables)
  DevBuf<int4> stencil;   // unpruned rows of a cell's stencil (k_tables)
  fx::Unit unit{};  // FP64 on the integer units, where unit.ok
};

void pair_layout_free(PairLayout *L) { delete L; }

// Workspace of a particle set's searches: a search builds its layout anew in
// buffers that only grow and go with the set.  One search at a time holds it, from
// the copy of host queries to the device on.
struct SearchSpace {
  std::mutex m;
  PairLayout L;
  HostStage queries;
  DevBuf<double> qsoa, dxd;
  DevBuf<int32_t> cnt, cols;
  DevBuf<int64_t> rowptr, rpk, sums;
  // Between searches it keeps what is in proportion to the set (about 80 B a
  // particle, and as much a query for no more queries than that) and lists up to
  // KEEP_BYTES; the buffers of a search with more queries, or longer lists, go back.
  void trim(int64_t nq, int64_t n) {
    if (nq > std::max(n, KEEP_QUERIES)) {
      L.rows_own.release();
      L.units.release(), L.singles.release(), L.exits.release();
      queries.buf.release(), qsoa.release(), cnt.release();
      rowptr.release(), rpk.release(), sums.release();
    }
    if (cols.cap * sizeof(int32_t) > KEEP_BYTES) cols.release();
    if (dxd.cap * sizeof(double) > KEEP_BYTES) dxd.release();
  }
  static constexpr int64_t KEEP_QUERIES = 1 << 20;
  static constexpr size_t KEEP_BYTES = size_t(256) << 20;
};
SearchSpace *search_space_new() { return new SearchSpace(); }
void search_space_free(SearchSpace *w) { delete w; }

namespace {

constexpr int TPB = 256;
constexpr int WARPS_PER_CTA = 4;
constexpr int GROUP_E2 = 4;  // a unit spans at most this many fine cells along e2
constexpr int COUNTS = 16;

enum { POL_COUNT = 0, POL_LIST = 1, POL_MATVEC = 2 };

// ------------------------------------------------------------ layout build ---
FineGrid make_fine_grid(const GridDesc &g, double r, int64_t npts, int F) {
  FineGrid fg{};
  fg.dim = g.dim;
  fg.eoff = 3 - g.dim;
  const double target = r > 0 ? r / F : 0.0;
  for (int e = 0; e < 3; ++e) {
    const int d = e - fg.eoff;
    if (d < 0) {
      fg.m[e] = 1;
      fg.h[e] = 1.0;
      fg.lo[e] = 0.0;
      fg.L[e] = 1.0;
      fg.periodic[e] = 0;
      continue;
    }
    fg.lo[e] = g.lo[d];
    fg.L[e] = g.hi[d] - g.lo[d];
    fg.periodic[e] = g.periodic[d];
    double m = target > 0 ? std::floor(fg.L[e] / target * (1.0 - 1e-9)) : 1.0;
    if (!(m >= 1.0)) m = 1.0;
    if (m > 1023.0) m = 1023.0;
    fg.m[e] = (int)m;
  }
  // keep the fine grid within a few cells per point
  const double cap = std::max<double>(64.0, 4.0 * (double)npts);
  for (int it = 0; it < 64; ++it) {
    double tot = (double)fg.m[0] * fg.m[1] * fg.m[2];
    if (tot <= cap) break;
    int eb = 0;
    for (int e = 1; e < 3; ++e)
      if (fg.m[e] > fg.m[eb]) eb = e;
    fg.m[eb] = std::max(1, (int)(fg.m[eb] * 0.8));
  }
  fg.ncells = (uint32_t)fg.m[0] * fg.m[1] * fg.m[2];
  for (int e = 0; e < 3; ++e) {
    const int d = e - fg.eoff;
    fg.h[e] = d < 0 ? 1.0 : fg.L[e] / fg.m[e];
    fg.hf[e] = (float)fg.h[e];
    fg.inv[e] = 1.0 / fg.h[e];
    fg.K[e] = d < 0 ? 0 : (int)std::ceil(r / fg.h[e] * (1.0 + 1e-9));
    if (fg.K[e] > 2 * fg.m[e] + 1) fg.K[e] = 2 * fg.m[e] + 1;
  }
  return fg;
}

// floor((x - lo) / h), unclamped; NaN: far outside, never a neighbour.  inv =
// 1 / h rounded: a coordinate on a cell boundary may land in the cell beside
// it, which the pruning margin (1e-9 of a cell) covers.  (A division here and
// in the layout made both kernels FP64-bound: 440 us each at N = 4M.)
__device__ __forceinline__ int fine_coord(double x, double lo, double inv) {
  const double t = (x - lo) * inv;
  if (!(fabs(t) < 1e9)) return t < 0.0 ? -1000000000 : 1000000000;
  return __double2int_rd(t);
}

// Sort key of a point: clamped fine cell (row-major, e2 fastest) times 8 plus
// its octant within the cell, so that consecutive points of a dense cell are
// also close together (tighter query tiles).
// blockIdx.y: the set (particles, queries).
struct PointSet {
  const double *src;  // SoA
  int64_t n, stride;
  int clamp;  // anchor cells clamped to the grid (k_fill_layout)
  uint32_t *keys;
  const uint32_t *perm;
  int4 *cell;
  float4 *loc;
  D4 *posk;
};
struct PointSets {
  PointSet s[2];
};
__global__ void k_fine_keys(PointSets sets, FineGrid fg) {
  const PointSet &S = sets.s[blockIdx.y];
  const double *__restrict__ src = S.src;
  const int64_t n = S.n, stride = S.stride;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c[3];
  uint32_t sub = 0;
  for (int e = 0; e < 3; ++e) {
    const int d = e - fg.eoff;
    if (d < 0) {
      c[e] = 0;
      continue;
    }
    const double x = src[(int64_t)d * stride + i];
    const int u = fine_coord(x, fg.lo[e], fg.inv[e]);
    c[e] = min(max(u, 0), fg.m[e] - 1);
    const double f = x - (fg.lo[e] + (double)c[e] * fg.h[e]);
    sub |= (f >= 0.5 * fg.h[e] ? 1u : 0u) << (2 - e);
  }
  S.keys[i] = ((((uint32_t)c[0] * fg.m[1] + c[1]) * fg.m[2] + c[2]) << 3) | sub;
}

// Anchor cell of a point: the clamped cell for column particles (their range
// membership), the unclamped cell for query points (which may lie outside
// the domain and must keep their true periodic image).  loc holds the FP32
// offset from the anchor cell's corner and, in .w, the anchor's e2 index as
// an (exact) float.
__global__ void k_fill_layout(PointSets sets, FineGrid fg) {
  const PointSet &S = sets.s[blockIdx.y];
  const double *__restrict__ src = S.src;
  const int64_t stride = S.stride;
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S.n) return;
  const uint32_t i = S.perm[k];
  double x[3];
  int u[3], c[3];
  float f[3];
  for (int e = 0; e < 3; ++e) {
    const int d = e - fg.eoff;
    if (d < 0) {
      x[e] = 0.0;
      u[e] = 0;
      c[e] = 0;
      f[e] = 0.f;
      continue;
    }
    x[e] = src[(int64_t)d * stride + i];
    u[e] = fine_coord(x[e], fg.lo[e], fg.inv[e]);
    c[e] = S.clamp ? min(max(u[e], 0), fg.m[e] - 1) : u[e];
    const double corner = fg.lo[e] + (double)c[e] * fg.h[e];
    f[e] = (float)(x[e] - corner);
  }
  S.cell[k] = make_int4(c[0], c[1], c[2], 0);
  S.loc[k] = make_float4(f[0], f[1], f[2], (float)c[2]);  // exact: c[2] < 2^24
  S.posk[k] = D4{x[0], x[1], x[2], 0.0};
}

// First index of keys[0, n) whose value is >= key, by a 32-way search (whole
// warps).
__device__ __forceinline__ int64_t warp_lower_bound(const uint32_t *__restrict__ keys, int64_t n,
                                                    uint64_t key, int lane) {
  int64_t lo = 0, hi = n;  // the answer lies in [lo, hi]
  while (hi - lo > 32) {
    const int64_t step = (hi - lo + 32) / 33;
    const int64_t i = lo + (int64_t)(lane + 1) * step;
    const unsigned m = __ballot_sync(0xffffffffu, i < hi && (uint64_t)keys[i < hi ? i : lo] < key);
    const int c = __popc(m);  // probes below the key form a prefix
    const int64_t nlo = c ? lo + (int64_t)c * step + 1 : lo;
    hi = c < 32 && lo + (int64_t)(c + 1) * step < hi ? lo + (int64_t)(c + 1) * step : hi;
    lo = nlo;
  }
  const unsigned m = __ballot_sync(0xffffffffu, lo + lane < hi && (uint64_t)keys[lo + lane] < key);
  return lo + __popc(m);
}

// cell_start[c] = first of the n sorted keys in cell c or beyond, c <= ncells:
// a CTA's cells are consecutive, so its threads search only between the first
// keys of its first and last cell, which two warps find.  (Marking, counting
// and scanning took six launches.)
__global__ void __launch_bounds__(TPB) k_cell_start(const uint32_t *__restrict__ keys, int64_t n,
                                                    uint32_t ncells,
                                                    uint32_t *__restrict__ cell_start) {
  __shared__ int64_t range[2];
  const int64_t c0 = (int64_t)blockIdx.x * TPB;
  const int w = threadIdx.x >> 5;
  if (w < 2) {
    const int64_t c = w ? min(c0 + TPB, (int64_t)ncells) : c0;
    const int64_t at = warp_lower_bound(keys, n, (uint64_t)c * 8, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0) range[w] = at;
  }
  __syncthreads();
  const int64_t c = c0 + threadIdx.x;
  if (c > (int64_t)ncells) return;
  int64_t lo = range[0], hi = range[1];
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((uint64_t)keys[mid] < (uint64_t)c * 8) lo = mid + 1; else hi = mid;
  }
  cell_start[c] = (uint32_t)lo;
}

// Fixed-point positions of a point set in kernel order.
__global__ void k_fill_fixed(const D4 *__restrict__ posk, int64_t n, fx::Unit U,
                             longlong2 *__restrict__ fxy, long long *__restrict__ fz) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const D4 x = posk[k];
  fxy[k] = make_longlong2(fx::to_fixed(x.x, U.f, U.k), fx::to_fixed(x.y, U.f, U.k));
  fz[k] = fx::to_fixed(x.z, U.f, U.k);
}

int reserve_points(int64_t n, const double *src_soa, int64_t stride, bool clamp_anchor,
                   PointLayout &P, PointSet &S) {
  P.n = n;
  ABX_TRY(P.perm.reserve(n ? n : 1));
  ABX_TRY(P.keys.reserve(n ? n : 1));
  ABX_TRY(P.cell.reserve(n ? n : 1));
  ABX_TRY(P.loc.reserve(n ? n : 1));
  ABX_TRY(P.posk.reserve(n ? n : 1));
  if (n) ABX_TRY(P.tmp.reserve(2 * (size_t)n + radix_temp_u32(n) + 64));
  S = PointSet{src_soa,    n,          stride,    clamp_anchor ? 1 : 0, P.keys.ptr,
               P.perm.ptr, P.cell.ptr, P.loc.ptr, P.posk.ptr};
  return ABX_OK;
}

// Kernel order of the particles and (rows) of the queries, which go through
// each launch together: at 100,000 each, separately, every launch left two
// thirds of the SMs idle.
int build_points(abx_context *ctx, PointSets &sets, PointLayout &cols, PointLayout *rows,
                 const FineGrid &fg) {
  cudaStream_t s = ctx->stream;
  const int64_t most = std::max(cols.n, rows ? rows->n : 0);
  if (most == 0) return ABX_OK;
  const dim3 grid(ceil_div(most, TPB), rows ? 2 : 1);
  k_fine_keys<<<grid, TPB, 0, s>>>(sets, fg);
  ABX_CHECK_CUDA(cudaGetLastError());
  int bits = 0;
  while (bits < 32 && (((uint64_t)fg.ncells * 8 - 1) >> bits) != 0) ++bits;
  SortSides S{};
  S.sides = rows ? 2 : 1;
  S.iota = true;
  for (int i = 0; i < S.sides; ++i) {
    PointLayout &P = i ? *rows : cols;
    S.s[i] = SortSide{P.keys.ptr, P.perm.ptr, P.tmp.ptr, P.tmp.ptr + P.n, P.tmp.ptr + 2 * P.n, (size_t)P.n};
  }
  ABX_TRY(radix_sort_sides(S, bits, s));
  k_fill_layout<<<grid, TPB, 0, s>>>(sets, fg);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

int build_cell_start(abx_context *ctx, PairLayout &L) {
  const uint32_t nc = L.fg.ncells;
  ABX_TRY(L.cell_start.reserve((size_t)nc + 1));
  k_cell_start<<<ceil_div((size_t)nc + 1, TPB), TPB, 0, ctx->stream>>>(L.cols.keys.ptr, L.cols.n, nc,
                                                                       L.cell_start.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

// Units: greedy runs of <= 32 consecutive queries (kernel order) whose anchor
// cells share (e0, e1) and span fewer than GROUP_E2 cells along e2.  One warp
// per (e0, e1) column walks its queries 32 at a time with the next 32 already
// loaded; the unit that starts at query s is the run of lanes that continue
// it.  A unit goes to the front of `units`, or, where `split` says so (low
// density, where a warp of 32 lanes would hold few queries), to the back, and
// its queries to `singles`, which k_pairs_thread walks.  Built on the host before,
// from a 16 B/point copy of the cells: 14 of the 39 ms of a search at N = 4M.
//
// Few columns (1-D: one) are walked by a warp per chunk of queries: where the first
// unit of a chunk starts depends on all before it, but is one of 32 places, from each
// of which a lane follows the chunk's units (k_unit_exits); going through the chunks
// with these answers is short (k_unit_entries).  A count of 1,000,000 points in 1-D:
// 13.2 ms with one warp, 1.0 so.
constexpr int UNIT_WARPS = 4;
constexpr uint32_t FEW_COLUMNS = 4;
constexpr int64_t MIN_CHUNK = 128, MOST_CHUNKS = 1024;

struct UnitQueries {
  const int4 *cell;
  const uint32_t *keys, *cell_start;
  bool self;
  int64_t n, chunk;  // queries a chunk
  int chunks;        // a column; 1: whole columns
  int m2;
};
// Queries of a column (whole warps).
__device__ __forceinline__ void column_range(const UnitQueries &Q, uint32_t col, int lane, int64_t &s,
                                             int64_t &end) {
  if (Q.self) {
    s = Q.cell_start[(uint64_t)col * Q.m2];
    end = Q.cell_start[(uint64_t)(col + 1) * Q.m2];
  } else {
    s = warp_lower_bound(Q.keys, Q.n, (uint64_t)col * Q.m2 * 8, lane);
    end = warp_lower_bound(Q.keys, Q.n, (uint64_t)(col + 1) * Q.m2 * 8, lane);
  }
}
// exits[item][e]: how far beyond the end of chunk `item` the units reach if one starts
// at its e-th query.
__global__ void __launch_bounds__(UNIT_WARPS * 32)
    k_unit_exits(UnitQueries Q, uint32_t items, uint8_t *__restrict__ exits) {
  const int lane = threadIdx.x & 31;
  const uint32_t item = blockIdx.x * UNIT_WARPS + (threadIdx.x >> 5);
  if (item >= items) return;
  int64_t s, end;
  column_range(Q, item / Q.chunks, lane, s, end);
  s += (int64_t)(item % Q.chunks) * Q.chunk;
  const int64_t stop = min(s + Q.chunk, end);
  s += lane;
  while (s < stop) {
    const int4 c0 = Q.cell[s];
    int run = 1;
    for (; run < 32 && s + run < end; ++run) {
      const int4 c = Q.cell[s + run];
      if (c.x != c0.x || c.y != c0.y || c.z < c0.z || c.z - c0.z >= GROUP_E2) break;
    }
    s += run;
  }
  exits[(size_t)item * 32 + lane] = (uint8_t)(s > stop ? min(s - stop, (int64_t)31) : 0);
}
// entries[item]: where the first unit of a chunk starts, from the chunk's first query.
__global__ void __launch_bounds__(32) k_unit_entries(int chunks, const uint8_t *__restrict__ exits,
                                                     uint8_t *__restrict__ entries) {
  const int lane = threadIdx.x;
  const size_t first = (size_t)blockIdx.x * chunks;
  int e = 0;
  for (int k0 = 0; k0 < chunks; k0 += 8) {
    int row[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) row[k] = k0 + k < chunks ? exits[(first + k0 + k) * 32 + lane] : 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (lane == 0 && k0 + k < chunks) entries[first + k0 + k] = (uint8_t)e;
      e = __shfl_sync(0xffffffffu, row[k], e);
    }
  }
}

__global__ void __launch_bounds__(UNIT_WARPS * 32)
    k_units(UnitQueries Q, const uint8_t *__restrict__ entries, FineGrid fg, int64_t cap, Split split,
            int2 *__restrict__ units, int *__restrict__ singles, int *__restrict__ counts) {
  const int lane = threadIdx.x & 31, m2 = fg.m[2], K2 = fg.K[2];
  const int4 *__restrict__ cell = Q.cell;
  const uint32_t *__restrict__ cell_start = Q.cell_start;
  const uint32_t items = (uint32_t)fg.m[0] * fg.m[1] * Q.chunks;
  const uint32_t warps = gridDim.x * UNIT_WARPS;
  for (uint32_t item = blockIdx.x * UNIT_WARPS + (threadIdx.x >> 5); item < items; item += warps) {
    const uint32_t col = item / Q.chunks;
    int64_t s, end;
    column_range(Q, col, lane, s, end);
    int64_t last = end;  // units start below it
    if (Q.chunks > 1) {
      s += (int64_t)(item % Q.chunks) * Q.chunk;
      last = min(s + Q.chunk, end);
      if (s >= end) continue;
      s += entries[item];
    }
    const int4 none = make_int4(0, 0, 0, 0);
    int64_t base = s;  // A holds queries [base, base + 32), B the 32 after them
    int4 A = base + lane < end ? cell[base + lane] : none;
    int4 B = base + 32 + lane < end ? cell[base + 32 + lane] : none;
    int2 mine = make_int2(0, 0);  // lane i keeps the i-th unit not written out yet
    int z_mine = 0;               // and its first cell along e2
    int held = 0;
    while (s < last || held > 0) {
      if (s < last) {
        if (s - base >= 32) {
          base += 32;
          A = B;
          B = base + 32 + lane < end ? cell[base + 32 + lane] : none;
        }
        const int o = (int)(s - base), src = (o + lane) & 31;
        const int ax = __shfl_sync(0xffffffffu, A.x, src), bx = __shfl_sync(0xffffffffu, B.x, src);
        const int ay = __shfl_sync(0xffffffffu, A.y, src), by = __shfl_sync(0xffffffffu, B.y, src);
        const int az = __shfl_sync(0xffffffffu, A.z, src), bz = __shfl_sync(0xffffffffu, B.z, src);
        const bool a = o + lane < 32;
        const int x = a ? ax : bx, y = a ? ay : by, z = a ? az : bz;
        const int x0 = __shfl_sync(0xffffffffu, x, 0), y0 = __shfl_sync(0xffffffffu, y, 0),
                  z0 = __shfl_sync(0xffffffffu, z, 0);
        const bool go = s + lane < end && x == x0 && y == y0 && z >= z0 && z - z0 < GROUP_E2;
        const unsigned stop = ~__ballot_sync(0xffffffffu, go);
        const int count = stop ? __ffs(stop) - 1 : 32;
        if (lane == held) {
          mine = make_int2((int)s, count);
          z_mine = z0;
        }
        ++held;
        s += count;
      }
      if (held == 32 || s >= last) {
        bool small = lane < held && mine.y < split.queries;
        if (small) {
          const int z = min(max(z_mine, 0), m2 - 1);
          const int za = max(z - K2, 0), zb = min(z + GROUP_E2 - 1 + K2, m2 - 1);
          const uint32_t *row = cell_start + (uint64_t)col * m2;
          small = row[zb + 1] - row[za] <= (uint32_t)split.row;
          if (split.around) {
            const int c0 = (int)(col / fg.m[1]), c1 = (int)(col % fg.m[1]);
            for (int o0 = -fg.K[0]; small && o0 <= fg.K[0]; ++o0)
              for (int o1 = -fg.K[1]; small && o1 <= fg.K[1]; ++o1) {
                int w0 = c0 + o0, w1 = c1 + o1;
                if (fg.periodic[0]) w0 += w0 < 0 ? fg.m[0] : w0 >= fg.m[0] ? -fg.m[0] : 0;
                if (fg.periodic[1]) w1 += w1 < 0 ? fg.m[1] : w1 >= fg.m[1] ? -fg.m[1] : 0;
                if (w0 < 0 || w0 >= fg.m[0] || w1 < 0 || w1 >= fg.m[1]) continue;
                const uint32_t *r = cell_start + ((uint64_t)w0 * fg.m[1] + w1) * m2;
                small = r[zb + 1] - r[za] <= (uint32_t)split.around;
              }
          }
        }
        const bool full = lane < held && !small;
        const unsigned mf = __ballot_sync(0xffffffffu, full), ms = __ballot_sync(0xffffffffu, small);
        const unsigned lt = (1u << lane) - 1u;
        int tot = small ? mine.y : 0, incl = tot;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane >= d) incl += v;
        }
        const int nsing = __shfl_sync(0xffffffffu, incl, 31);
        int bf = 0, bs = 0, bq = 0;
        if (lane == 0) {
          if (mf) bf = atomicAdd(&counts[0], __popc(mf));
          if (ms) {
            bs = atomicAdd(&counts[1], __popc(ms));
            bq = atomicAdd(&counts[2], nsing);
          }
        }
        bf = __shfl_sync(0xffffffffu, bf, 0);
        bs = __shfl_sync(0xffffffffu, bs, 0);
        bq = __shfl_sync(0xffffffffu, bq, 0);
        if (full) units[bf + __popc(mf & lt)] = mine;
        if (small) {
          units[cap - 1 - (bs + __popc(ms & lt))] = mine;
          for (int k = 0; k < mine.y; ++k) singles[bq + incl - tot + k] = mine.x + k;
        }
        held = 0;
      }
    }
  }
}

int build_units(abx_context *ctx, PairLayout &L, const Split &split) {
  PointLayout &Q = *L.rows;
  L.split = split;
  const int64_t n = Q.n;
  ABX_REQUIRE(n < (int64_t)0x7fffffff, ABX_ERR_INVALID, "too many query points");
  ABX_TRY(L.units.reserve(n ? n : 1));
  ABX_TRY(L.singles.reserve(n ? n : 1));
  ABX_TRY(L.counts.reserve(COUNTS));
  ABX_CHECK_CUDA(cudaMemsetAsync(L.counts.ptr, 0, COUNTS * sizeof(int), ctx->stream));
  if (n == 0) return ABX_OK;
  const uint32_t ncol = (uint32_t)L.fg.m[0] * L.fg.m[1];
  UnitQueries U{Q.cell.ptr, Q.keys.ptr, L.cell_start.ptr, L.self, n, n, 1, L.fg.m[2]};
  if (ncol <= FEW_COLUMNS && n > MIN_CHUNK) {
    U.chunk = std::max(MIN_CHUNK, (n / MOST_CHUNKS + 32) / 32 * 32);
    U.chunks = (int)ceil_div(n, U.chunk);
    const uint32_t items = ncol * U.chunks;
    ABX_TRY(L.exits.reserve((size_t)items * 33));
    uint8_t *entries = L.exits.ptr + (size_t)items * 32;
    k_unit_exits<<<ceil_div(items, UNIT_WARPS), UNIT_WARPS * 32, 0, ctx->stream>>>(U, items, L.exits.ptr);
    k_unit_entries<<<ncol, 32, 0, ctx->stream>>>(U.chunks, L.exits.ptr, entries);
  }
  const uint32_t items = ncol * U.chunks;
  const unsigned blocks = std::min(ceil_div(items, UNIT_WARPS), 8u * (unsigned)ctx->num_sms);
  k_units<<<blocks, UNIT_WARPS * 32, 0, ctx->stream>>>(
      U, U.chunks > 1 ? L.exits.ptr + (size_t)items * 32 : nullptr, L.fg, n, split, L.units.ptr,
      L.singles.ptr, L.counts.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

// ------------------------------------------------------------- kernels ---
constexpr int EXT_TAB = 64;   // extent table covers gaps of < 64 cells in e0, e1
constexpr int SEG_CAP = 96;   // segments per batch (32 rows x up to 3 image splits)

struct KParams {
  FineGrid fg;
  double r, r2;
  double prune2;  // squared pruning distance (r plus a safety margin)
  // radius-search norm: 2 euclidean, 1 manhattan, -1 chebyshev (the
  // reference's distance_helper<2/1/-1>); thr = get_value_to_accumulate(r)
  int lnorm;
  double thr;
  const int *ext;  // [EXT_TAB*EXT_TAB]: max e2 gap (cells) for e0/e1 gaps, -1 pruned
  // kernel functor parameters
  int kind;
  double p0;
  float p0f, c_exp2;  // c_exp2 = -p0*log2(e)
  // columns (kernel order)
  const float4 *cloc;
  const D4 *cpos;
  const uint32_t *cell_start;
  const float *b32;
  const double *b64;
  const double *s_col;
  // queries (kernel order)
  const int4 *qcell;
  const float4 *qloc;
  const D4 *qpos;
  const double *s_row;
  const int2 *units;     // full units from the front, small ones from the back
  int64_t units_cap;
  const int *singles;    // queries of the small units
  const int *counts;     // full units, small units, singles
  int all_units;         // 1: the small units too (searches that write lists)
  int *counter;          // work counters: units, singles
  UnitWork work;         // of the two kernels, as far as the host knows
  const float4 *bands;   // two entries a span: r2lo, r2hi, r2box, rbox_inf; r2mid, r2half
  const int4 *stencil;   // unpruned rows of a cell's stencil, counts[3] of them
  int lanes;             // lanes a query of the singles
  int self;              // the queries are the columns, in the same order
  float near2;           // Laplace in fixed point: pairs closer than its root go by FP64
  // fixed point (fix64.cuh): column and query positions, box lengths, constants
  const longlong2 *fxy, *qfxy;
  const long long *fz, *qfz;
  long long Lfix[3];
  fx::Consts fixc;
  // outputs (by row)
  int32_t *counts_out;
  const int64_t *rowptr;  // for LIST: query kernel order -> output offset
  int32_t *cols_out;      // storage index of the column particle
  double *dx_out;         // for LIST (optional): x_j - (x_i + image*L), D per pair
  const uint32_t *cperm;  // column kernel order -> storage index
  const uint32_t *qperm;  // query kernel order -> row
  double *c;
};

// Hardware base-2 exponential (MUFU, ~2 ulp), flush-to-zero: the kernel
// weights it serves are negligible long before 2^-126.
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <int KIND> __device__ __forceinline__ float kern32(float d2, const KParams &P) {
  if (KIND == ABX_K_CONST) return P.p0f;
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return ex2_approx(d2 * P.c_exp2);
  if (KIND == ABX_K_WENDLAND_C2) {
    const float q = d2 * rsqrtf(fmaxf(d2, 1e-36f)) * P.p0f;
    const float t = fmaxf(1.0f - q, 0.0f);
    const float t2 = t * t;
    return t2 * t2 * fmaf(4.0f, q, 1.0f);
  }
  if (KIND == ABX_K_LAPLACE) return __fdividef(1.0f, d2 * rsqrtf(fmaxf(d2, 1e-36f)) + P.p0f);
  if (KIND == ABX_K_MULTIQUADRIC) {
    const float a = d2 + P.p0f;
    return a * rsqrtf(fmaxf(a, 1e-36f));
  }
  return 0.f;
}

template <int KIND>
__device__ __forceinline__ double kern64(double d2, const KParams &P, double si, double sj) {
  if (KIND == ABX_K_CONST) return P.p0;
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return exp(-d2 * P.p0);
  if (KIND == ABX_K_WENDLAND_C2) {
    const double q = sqrt(d2) * P.p0;
    if (q >= 1.0) return 0.0;
    const double t = 1.0 - q;
    const double t2 = t * t;
    return t2 * t2 * (4.0 * q + 1.0);
  }
  if (KIND == ABX_K_LAPLACE) return 1.0 / (sqrt(d2) + P.p0);
  if (KIND == ABX_K_MULTIQUADRIC) return sqrt(d2 + P.p0);
  if (KIND == ABX_K_SCALAR_SUM) return si + sj;
  return 0.0;
}

// The reference's FP64 acceptance test for one (query, candidate, image):
// accum = ((0 + dx0^2) + dx1^2) + dx2^2 over the REAL dimensions in order, no
// FMA, with dx = x_j - (x_i + image*L); inside iff !(accum > r^2).
__device__ __forceinline__ double exact_d2(const D4 &xq, const D4 &xj, const int *img,
                                           const FineGrid &fg) {
  const double q[3] = {xq.x, xq.y, xq.z};
  const double p[3] = {xj.x, xj.y, xj.z};
  double acc = 0.0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (e < fg.eoff) continue;
    const double cur = __dadd_rn(q[e], __dmul_rn((double)img[e], fg.L[e]));
    const double dx = __dsub_rn(p[e], cur);
    acc = __dadd_rn(acc, __dmul_rn(dx, dx));
  }
  return acc;
}

// The reference's test in the manhattan and chebyshev norms
// (distance_helper<1>, <-1>, src/detail/Distance.h:46-137): accum starts at 0
// and takes |dx| over the real dimensions in order, summed (1) or as a running
// maximum (-1); inside iff !(accum > |r|).
__device__ __forceinline__ double exact_norm(const D4 &xq, const D4 &xj, const int *img,
                                             const FineGrid &fg, int lnorm) {
  if (lnorm == 2) return exact_d2(xq, xj, img, fg);
  const double q[3] = {xq.x, xq.y, xq.z};
  const double p[3] = {xj.x, xj.y, xj.z};
  double acc = 0.0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (e < fg.eoff) continue;
    const double cur = __dadd_rn(q[e], __dmul_rn((double)img[e], fg.L[e]));
    const double a = fabs(__dsub_rn(p[e], cur));
    if (lnorm == 1)
      acc = __dadd_rn(acc, a);
    else if (a > acc)
      acc = a;
  }
  return acc;
}

__device__ __forceinline__ void unpack_seg(int z, int img[3], int &du0, int &du1) {
  img[0] = (z & 3) - 1;
  img[1] = ((z >> 2) & 3) - 1;
  img[2] = ((z >> 4) & 3) - 1;
  du0 = ((z >> 6) & 0xfff) - 2048;
  du1 = ((z >> 18) & 0xfff) - 2048;
}

constexpr int CENTRE = 21;  // the image bits of a segment (and of `code`): 0 in every dimension

// dx of an accepted pair as the reference's search iterator exposes it:
// x_j - (x_i + image*L) over the real dimensions (src/Search.h:188-190, 443),
// written as D doubles at pair slot `slot`.
__device__ __forceinline__ void write_dx(const KParams &P, int64_t slot, const D4 &xq, int k,
                                         int seg_z) {
  const FineGrid &fg = P.fg;
  int img[3], du0, du1;
  unpack_seg(seg_z, img, du0, du1);
  const D4 xj = P.cpos[k];
  const double q[3] = {xq.x, xq.y, xq.z};
  const double p[3] = {xj.x, xj.y, xj.z};
  const int D = 3 - fg.eoff;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (e < fg.eoff) continue;
    const double cur = __dadd_rn(q[e], __dmul_rn((double)img[e], fg.L[e]));
    P.dx_out[slot * D + (e - fg.eoff)] = __dsub_rn(p[e], cur);
  }
}

// Per-warp shared state: the segment list of one batch of rows, its length
// prefix, and one staged tile of candidates.
struct WarpSeg {
  int4 seg[SEG_CAP];      // start, end, packed(img, du0, du1), c2shift
  float4 segf[SEG_CAP];   // du0, du1, c2shift as exact floats (staging offsets)
  int off[SEG_CAP + 1];   // exclusive prefix of segment lengths
};

// Build the candidate segments of rows [row0, row0+32) of the unit's stencil
// into ws.seg (warp-cooperative: one row per lane, up to three image splits
// along e2).  Returns the number of segments; ws.off holds the length prefix.
__device__ __forceinline__ int build_segments(const KParams &P, const int lo[3], const int hi[3],
                                              int a0, int a1, int R1, int nrows, int row0,
                                              WarpSeg &ws, int lane) {
  const FineGrid &fg = P.fg;
  int4 mine[3];
  bool has[3] = {false, false, false};
  const int t = row0 + lane;
  int u0s = 0, u1s = 0;
  if (t < nrows) {
    const int u0 = a0 + t / R1, u1 = a1 + t % R1;
    u0s = u0;
    u1s = u1;
    const int g0c = max(max(lo[0] - u0, u0 - hi[0]) - 1, 0);
    const int g1c = max(max(lo[1] - u1, u1 - hi[1]) - 1, 0);
    int ext;
    if (P.lnorm == -1) {
      // the chebyshev ball is the whole stencil box: no euclidean pruning
      ext = fg.K[2];
    } else if (g0c < EXT_TAB && g1c < EXT_TAB) {
      // euclidean pruning also serves the manhattan ball, which lies inside
      ext = P.ext[g0c * EXT_TAB + g1c];
    } else {
      const double g0 = g0c * fg.h[0], g1 = g1c * fg.h[1];
      const double rem = P.prune2 - g0 * g0 - g1 * g1;
      ext = rem < 0.0 ? -1 : min((int)floor(sqrt(rem) / fg.h[2]), fg.K[2]);
    }
    if (ext >= 0) {
      int w0 = u0, i0 = 0, w1 = u1, i1 = 0;
      if (u0 < 0) { w0 = u0 + fg.m[0]; i0 = 1; } else if (u0 >= fg.m[0]) { w0 = u0 - fg.m[0]; i0 = -1; }
      if (u1 < 0) { w1 = u1 + fg.m[1]; i1 = 1; } else if (u1 >= fg.m[1]) { w1 = u1 - fg.m[1]; i1 = -1; }
      const int a2 = max(lo[2] - 1 - ext, lo[2] - fg.K[2]);
      const int b2 = min(hi[2] + 1 + ext, hi[2] + fg.K[2]);
      const uint32_t rowbase = ((uint32_t)w0 * fg.m[1] + w1) * (uint32_t)fg.m[2];
      const int m2 = fg.m[2];
#pragma unroll
      for (int sgi = 0; sgi < 3; ++sgi) {
        if (sgi != 1 && !fg.periodic[2]) continue;
        const int slo = sgi == 0 ? -m2 : (sgi == 1 ? 0 : m2);
        const int shi = sgi == 0 ? -1 : (sgi == 1 ? m2 - 1 : 2 * m2 - 1);
        const int sa = max(a2, slo), sb = min(b2, shi);
        if (sa > sb) continue;
        const int i2 = 1 - sgi;            // image +1, 0, -1
        const int shift = i2 * m2;         // wrapped w2 = u2 + shift
        const uint32_t start = P.cell_start[rowbase + (uint32_t)(sa + shift)];
        const uint32_t end = P.cell_start[rowbase + (uint32_t)(sb + shift) + 1];
        if (start >= end) continue;
        const int z = (i0 + 1) | ((i1 + 1) << 2) | ((i2 + 1) << 4) |
                      ((u0 - lo[0] + 2048) << 6) | ((u1 - lo[1] + 2048) << 18);
        mine[sgi] = make_int4((int)start, (int)end, z, -shift - lo[2]);
        has[sgi] = true;
      }
    }
  }
  // compact into the shared list
  const unsigned lt = (1u << lane) - 1u;
  int base = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned m = __ballot_sync(0xffffffffu, has[k]);
    if (has[k]) {
      const int slot = base + __popc(m & lt);
      ws.seg[slot] = mine[k];
      ws.segf[slot] = make_float4((float)(u0s - lo[0]), (float)(u1s - lo[1]), (float)mine[k].w, 0.f);
    }
    base += __popc(m);
  }
  __syncwarp();
  // exclusive prefix of the lengths: lane l owns entries 3l..3l+2
  int len[3], s = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = 3 * lane + k;
    len[k] = i < base ? ws.seg[i].y - ws.seg[i].x : 0;
    s += len[k];
  }
  int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int run = incl - s;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = 3 * lane + k;
    if (i < base) ws.off[i] = run;
    run += len[k];
  }
  if (lane == 31) ws.off[base] = run;  // total
  __syncwarp();
  return base;
}

constexpr int STAGE = 64;  // candidates staged per round (two per lane)

// Internal kernel tag: Wendland C2 in a mixed-precision matvec whose kernel
// support 1/p0 is no larger than the search radius (p0 * r >= 1 - 1e-9).  The kernel
// then vanishes at and beyond the cut-off to fourth order, so the clamp
// max(1 - q, 0) is the whole cut-off test: a pair whose FP32 and FP64
// classifications differ has |q - 1| <= delta with delta ~ 1e-5 (the FP32
// rounding band of d^2 relative to r^2), and contributes at most
// 5 delta^4 |b_j| < 1e-19 |b_j| either way -- far below the FP32 term
// precision -- so no pair needs the exact FP64 re-test.  Coordinates are
// staged pre-scaled by p0, making d^2 = q^2 directly.
constexpr int K_WEND_CUT = 100 + ABX_K_WENDLAND_C2;

struct WarpTile32 {
  float4 p[STAGE];
  // the same candidates as pairs for the packed FP32x2 loop:
  // pp[2h] = (x_a, x_b, y_a, y_b), pp[2h+1] = (z_a, z_b, b_a, b_b), a = 2h, b = 2h+1
  float4 pp[STAGE + 2];
  int2 meta[STAGE];  // column kernel index, segment index
};

// Hardware reciprocal square root (MUFU, ~2 ulp), flush-to-zero: callers
// keep x >= 1e-30 so that no denormal or zero reaches it.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Kernel values of two pairs at once on the packed FP32x2 pipe.
template <int KIND> __device__ __forceinline__ float2 kern32x2(float2 dd, const KParams &P) {
  if (KIND == ABX_K_CONST) return make_float2(P.p0f, P.p0f);
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) {
    const float2 e = __fmul2_rn(dd, make_float2(P.c_exp2, P.c_exp2));
    return make_float2(ex2_approx(e.x), ex2_approx(e.y));
  }
  const float2 r = make_float2(sqrt_approx(dd.x), sqrt_approx(dd.y));
  if (KIND == ABX_K_WENDLAND_C2) {
    const float2 q = __fmul2_rn(r, make_float2(P.p0f, P.p0f));
    const float2 t = __ffma2_rn(q, make_float2(-1.f, -1.f), make_float2(1.f, 1.f));
    const float2 t2 = __fmul2_rn(t, t);
    const float2 t4 = __fmul2_rn(t2, t2);
    const float2 pw = __ffma2_rn(q, make_float2(4.f, 4.f), make_float2(1.f, 1.f));
    return __fmul2_rn(t4, pw);
  }
  if (KIND == ABX_K_LAPLACE) {
    const float2 a = __fadd2_rn(r, make_float2(P.p0f, P.p0f));
    return make_float2(__fdividef(1.f, a.x), __fdividef(1.f, a.y));
  }
  if (KIND == ABX_K_MULTIQUADRIC) {
    const float2 a = __fadd2_rn(dd, make_float2(P.p0f, P.p0f));
    return make_float2(sqrt_approx(a.x), sqrt_approx(a.y));
  }
  return make_float2(0.f, 0.f);
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Unit prologue shared by both kernels: the warp's anchor-cell box [lo, hi]
// and the row range of its stencil.
__device__ __forceinline__ void unit_box(const KParams &P, const int4 qc, bool active, int lo[3],
                                         int hi[3], int &a0, int &a1, int &R1, int &nrows) {
  const FineGrid &fg = P.fg;
  lo[0] = hi[0] = qc.x;
  lo[1] = hi[1] = qc.y;
  lo[2] = hi[2] = qc.z;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const int a = active ? lo[e] : 0x7fffffff, b = active ? hi[e] : -0x7fffffff;
    lo[e] = __reduce_min_sync(0xffffffffu, a);
    hi[e] = __reduce_max_sync(0xffffffffu, b);
  }
  a0 = max(lo[0] - fg.K[0], fg.periodic[0] ? -fg.m[0] : 0);
  const int b0 = min(hi[0] + fg.K[0], fg.periodic[0] ? 2 * fg.m[0] - 1 : fg.m[0] - 1);
  a1 = max(lo[1] - fg.K[1], fg.periodic[1] ? -fg.m[1] : 0);
  const int b1 = min(hi[1] + fg.K[1], fg.periodic[1] ? 2 * fg.m[1] - 1 : fg.m[1] - 1);
  R1 = b1 - a1 + 1;
  const int R0 = b0 - a0 + 1;
  nrows = (R0 > 0 && R1 > 0) ? R0 * R1 : 0;
}

// Rounding band of a tile whose FP32 offsets reach `span` cells from their
// reference corner: an offset carries < (3*span+2)*h*2^-24 error and a
// difference of two < edx = (span+2)*h*2^-20; |d2_f32 - d2| <= band.
struct TileBand {
  float4 a;  // r2lo, r2hi: accepted up to r2lo, rejected beyond r2hi; r2box, rbox_inf
  float4 b;  // r2mid, r2half: the band as |d2 - r2mid| <= r2half
};
constexpr int BAND_TAB = 64;
__device__ __forceinline__ TileBand tile_band(int span, const FineGrid &fg, double r, double r2,
                                              double thr, int norm) {
  const double hmax = fmax(fmax(fg.h[0] * (fg.eoff <= 0), fg.h[1] * (fg.eoff <= 1)), fg.h[2]);
  const double edx = (double)(span + 2) * hmax * 9.5367431640625e-07;
  const double band = 2.0 * 1.7320508075688772 * (r + edx) * edx + 3.0 * edx * edx +
                      4.0 * 5.960464477539063e-08 * r2 + 1e-300;
  // manhattan / chebyshev: each FP32 |d_e| is within edx of the exact one,
  // the sum of three adds <= 2 roundings of a value below 3 r
  const double nband = norm == 1 ? 3.0 * edx + 6.0 * 5.960464477539063e-08 * 3.0 * r + 1e-300
                                 : edx + 2.0 * 5.960464477539063e-08 * r + 1e-300;
  // (when the band reaches below 0 nothing is accepted outright: two
  // distinct points may share an FP32 offset, d = 0, yet lie outside a
  // radius smaller than the band)
  const double lo_thr = norm == 2 ? r2 - band : thr - nband;
  const float r2lo = lo_thr > 0.0 ? __double2float_rd(lo_thr) : -1.0f;
  const float r2hi = norm == 2 ? __double2float_ru(r2 + band) : __double2float_ru(thr + nband);
  // box test: euclidean for norms 2 and 1 (the manhattan ball lies inside
  // the euclidean one), a max-norm test for the chebyshev ball
  const float r2box = __double2float_ru((r2 + band) * (1.0 + 1e-6) + 1e-300);
  const float rbox_inf = __double2float_ru((thr + nband) * (1.0 + 1e-6) + 1e-300);
  // the band around its middle, widened by a few ulps so that the FP32
  // subtraction never shrinks it below (r2lo, r2hi]
  const float r2mid = (float)(0.5 * ((double)r2lo + (double)r2hi));
  const float r2half =
      __double2float_ru(0.5 * ((double)r2hi - (double)r2lo) + 8.0 * 5.960464477539063e-08 * r2);
  return {make_float4(r2lo, r2hi, r2box, rbox_inf), make_float4(r2mid, r2half, 0.f, 0.f)};
}

// Largest e2 gap (in cells) that keeps a cell within the pruning distance, for
// every pair of e0/e1 gaps below EXT_TAB cells (-1: pruned), and the bands by
// span: ~30 FP64 operations a unit otherwise, 0.4 of a unit's time where it
// holds few queries.
//
// rows: the rows (e0, e1 offsets) of a single cell's stencil that are not
// pruned, in row-major order, as (o0, o1, reach along e2); their number goes
// to counts[3] (k_pairs_thread).  By block 0, which also decides whether the
// small units are worked by the unit kernel after all and tells the host which
// of the two kernels have work.
constexpr int TABLE_TPB = 256;
constexpr int ROWS_MAX = 1024;  // (2 K0 + 1)(2 K1 + 1), K <= 7 (make_fine_grid)
__device__ __forceinline__ int row_reach(int a, int b, const FineGrid &fg, double prune2, int norm) {
  if (norm == -1) return fg.K[2];  // the chebyshev ball is the whole stencil box
  const int g0c = max(abs(a) - 1, 0), g1c = max(abs(b) - 1, 0);
  const double g0 = g0c * fg.h[0], g1 = g1c * fg.h[1];
  const double rem = __dsub_rn(__dsub_rn(prune2, __dmul_rn(g0, g0)), __dmul_rn(g1, g1));
  return rem < 0.0 ? -1 : min((int)fmin(floor(sqrt(rem) / fg.h[2]), (double)fg.K[2]) + 1, fg.K[2]);
}
__global__ void __launch_bounds__(TABLE_TPB) k_tables(FineGrid fg, double prune2, double r,
                                                      double thr, int norm, int *__restrict__ ext,
                                                      float4 *__restrict__ bands,
                                                      int4 *__restrict__ rows,
                                                      int *__restrict__ counts, int nq, int fold_at,
                                                      uint64_t *work, uint32_t seq) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x == 0) {
    __shared__ int wsum[TABLE_TPB / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int R1 = 2 * fg.K[1] + 1, NR = (2 * fg.K[0] + 1) * R1;
    int done = 0;
    for (int i0 = 0; i0 < NR; i0 += TABLE_TPB) {
      const int i = i0 + threadIdx.x;
      const int a = i / R1 - fg.K[0], b = i % R1 - fg.K[1];
      const int reach = i < NR ? row_reach(a, b, fg, prune2, norm) : -1;
      const unsigned m = __ballot_sync(0xffffffffu, reach >= 0);
      if (lane == 0) wsum[w] = __popc(m);
      __syncthreads();
      int at = done + __popc(m & ((1u << lane) - 1u));
      for (int k = 0; k < TABLE_TPB / 32; ++k) {
        if (k < w) at += wsum[k];
        done += wsum[k];
      }
      if (reach >= 0 && at < ROWS_MAX) rows[at] = make_int4(a, b, reach, 0);
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      counts[3] = min(done, ROWS_MAX);
      // a second kernel is not worth its launch for few queries
      const bool fold = (int64_t)counts[2] * fold_at < nq;
      counts[8] = fold ? counts[1] : 0;
      counts[9] = fold ? 0 : counts[2];
      if (work)
        *(volatile uint64_t *)work = unit_work_word(seq, counts[0] + counts[8] > 0, counts[9] > 0);
    }
  }
  if (t < EXT_TAB * EXT_TAB) {
    const double g0 = (t / EXT_TAB) * fg.h[0], g1 = (t % EXT_TAB) * fg.h[1];
    const double rem = __dsub_rn(__dsub_rn(prune2, __dmul_rn(g0, g0)), __dmul_rn(g1, g1));
    ext[t] = rem < 0.0 ? -1 : (int)fmin(floor(sqrt(rem) / fg.h[2]), (double)fg.K[2]);
  }
  if (t < BAND_TAB) {
    const TileBand b = tile_band(t, fg, r, r * r, thr, norm);
    bands[2 * t] = b.a;
    bands[2 * t + 1] = b.b;
  }
}

// Mixed-precision pair kernel.  Per unit (one warp, <= 32 queries):
//   rows of the stencil -> segment list -> flattened candidate stream, 32 at a
//   time -> each lane stages one candidate (FP32 offset from the unit's
//   reference corner) and keeps it only if it lies within r of the warp's
//   query bounding box -> every lane tests its query against the kept
//   candidates.  Pairs with d2 <= r2lo are accepted in the branch-free loop;
//   pairs in the rounding band (r2lo, r2hi] are re-decided afterwards with the
//   exact FP64 test, which is rare enough to run divergently.
// FP32 distance of a staged pair in the search norm (2: squared euclidean,
// 1: manhattan, -1: chebyshev), compared against the FP32 thresholds.
template <int NORM> __device__ __forceinline__ float norm32(float d0, float d1, float d2) {
  if (NORM == 1) return fabsf(d0) + fabsf(d1) + fabsf(d2);
  if (NORM == -1) return fmaxf(fabsf(d0), fmaxf(fabsf(d1), fabsf(d2)));
  return fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
}

template <int POL, int KIND, int NORM = 2>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32, 7)
    k_pairs_mixed(KParams P) {
  static_assert(NORM == 2 || POL != POL_MATVEC, "matvecs use the euclidean distance");
  __shared__ WarpSeg seg_all[WARPS_PER_CTA];
  __shared__ WarpTile32 tile_all[WARPS_PER_CTA];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpSeg &ws = seg_all[wid];
  WarpTile32 &sm = tile_all[wid];
  const FineGrid &fg = P.fg;
  const unsigned lt = (1u << lane) - 1u;
  constexpr bool WCUT = KIND == K_WEND_CUT;
  constexpr bool PCOUNT = POL == POL_COUNT && NORM == 2;  // counts two candidates at a time
  const float sc = WCUT ? P.p0f : 1.f;  // staging scale (d^2 = q^2 for WCUT)
  const int nfull = P.counts[0], nunits = nfull + P.counts[P.all_units ? 1 : 8];
  if (blockIdx.x * WARPS_PER_CTA >= nunits) return;  // see grid_blocks
  for (;;) {
    int unit = 0;
    if (lane == 0) unit = atomicAdd(P.counter, 1);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (unit >= nunits) break;
    const int2 U = unit < nfull ? P.units[unit] : P.units[P.units_cap - 1 - (unit - nfull)];
    const bool active = lane < U.y;
    const int qi = U.x + (active ? lane : 0);
    const int4 qc = P.qcell[qi];
    const float4 ql = P.qloc[qi];
    int lo[3], hi[3], a0, a1, R1, nrows;
    unit_box(P, qc, active, lo, hi, a0, a1, R1, nrows);
    const float pq0 = fmaf((float)(qc.x - lo[0]), fg.hf[0], ql.x);
    const float pq1 = fmaf((float)(qc.y - lo[1]), fg.hf[1], ql.y);
    const float pq2 = fmaf((float)(qc.z - lo[2]), fg.hf[2], ql.z);
    // warp bounding box of the query offsets (inactive lanes repeat lane 0)
    const float bl0 = warp_min(pq0), bh0 = warp_max(pq0);
    const float bl1 = warp_min(pq1), bh1 = warp_max(pq1);
    const float bl2 = warp_min(pq2), bh2 = warp_max(pq2);
    // the box as centre and half-width, the half-width rounded outwards (a
    // wider box only keeps more candidates; none within r is dropped)
    const float bc0 = 0.5f * (bl0 + bh0), bw0 = __fadd_ru(0.5f * (bh0 - bl0), 1e-6f * (fabsf(bl0) + fabsf(bh0)));
    const float bc1 = 0.5f * (bl1 + bh1), bw1 = __fadd_ru(0.5f * (bh1 - bl1), 1e-6f * (fabsf(bl1) + fabsf(bh1)));
    const float bc2 = 0.5f * (bl2 + bh2), bw2 = __fadd_ru(0.5f * (bh2 - bl2), 1e-6f * (fabsf(bl2) + fabsf(bh2)));
    // rounding band: every staged coordinate lies within `span` cells of the
    // reference corner (tile_band)
    int span = 0;
#pragma unroll
    for (int e = 0; e < 3; ++e) span = max(span, hi[e] - lo[e] + 2 * fg.K[e] + 2);
    const TileBand bd = span < BAND_TAB ? TileBand{P.bands[2 * span], P.bands[2 * span + 1]}
                                        : tile_band(span, fg, P.r, P.r2, P.thr, NORM);
    const float r2lo = bd.a.x, r2hi = bd.a.y, r2box = bd.a.z, rbox_inf = bd.a.w;
    const float r2mid = bd.b.x, r2half = bd.b.y;
    D4 xq;
    bool have_xq = false;
    double acc64 = 0.0;
    int count = 0;
    int64_t out_off = 0;
    if (POL == POL_LIST && active) out_off = P.rowptr[qi];
    if (POL == POL_LIST && P.dx_out) {
      xq = P.qpos[qi];
      have_xq = true;
    }

    for (int row0 = 0; row0 < nrows; row0 += 32) {
      const int nseg = build_segments(P, lo, hi, a0, a1, R1, nrows, row0, ws, lane);
      if (nseg == 0) continue;
      const int total = ws.off[nseg];
      int cur = 0;  // this lane's segment; its candidate index only grows
      for (int t0 = 0; t0 < total; t0 += STAGE) {
        int nt = 0;
        // staging in three phases so that the global loads of every
        // sub-round are in flight together: (1) candidate indices from the
        // segment list, (2) positions and weights, (3) bounding-box test and
        // compaction into shared memory
        constexpr int NS = STAGE / 32;
        int kk[NS], sx[NS];
        float4 so[NS];
#pragma unroll
        for (int sub = 0; sub < NS; ++sub) {
          const int t = t0 + sub * 32 + lane;
          kk[sub] = -1;
          sx[sub] = 0;
          so[sub] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (t < total) {
            while (cur + 1 < nseg && ws.off[cur + 1] <= t) ++cur;
            sx[sub] = cur;
            kk[sub] = ws.seg[cur].x + (t - ws.off[cur]);
            so[sub] = ws.segf[cur];
          }
        }
        float4 cls[NS];
        float bws[NS];
#pragma unroll
        for (int sub = 0; sub < NS; ++sub) {
          cls[sub] = make_float4(0.f, 0.f, 0.f, 0.f);
          bws[sub] = 0.f;
          if (kk[sub] >= 0) {
            cls[sub] = __ldg(&P.cloc[kk[sub]]);
            if (POL == POL_MATVEC) bws[sub] = __ldg(&P.b32[kk[sub]]);
            if (POL == POL_LIST) bws[sub] = __uint_as_float(__ldg(&P.cperm[kk[sub]]));
          }
        }
#pragma unroll
        for (int sub = 0; sub < NS; ++sub) {
          bool keep = false;
          float4 st;
          const int k = kk[sub], sidx = sx[sub];
          if (k >= 0) {
            const float4 cl = cls[sub];
            // offsets from the unit's reference corner: whole cells (exact
            // small integers) times the cell size plus the in-cell offset
            st.x = fmaf(so[sub].x, fg.hf[0], cl.x);
            st.y = fmaf(so[sub].y, fg.hf[1], cl.y);
            st.z = fmaf(cl.w + so[sub].z, fg.hf[2], cl.z);
            const float e0 = fmaxf(fabsf(st.x - bc0) - bw0, 0.f);
            const float e1 = fmaxf(fabsf(st.y - bc1) - bw1, 0.f);
            const float e2 = fmaxf(fabsf(st.z - bc2) - bw2, 0.f);
            keep = NORM == -1 ? fmaxf(e0, fmaxf(e1, e2)) <= rbox_inf
                              : fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) <= r2box;
            st.w = bws[sub];
          }
          const unsigned km = __ballot_sync(0xffffffffu, keep);
          if (WCUT) {
            // natural order, one 16-byte store per lane (no bank conflicts);
            // repacked into candidate pairs below
            if (keep) sm.p[nt + __popc(km & lt)] = make_float4(st.x * sc, st.y * sc, st.z * sc, st.w);
          } else if (keep) {
            const int slot = nt + __popc(km & lt);
            sm.p[slot] = st;
            sm.meta[slot] = make_int2(k, sidx);
            if (POL == POL_MATVEC) {
              float *pf = reinterpret_cast<float *>(&sm.pp[2 * (slot >> 1)]);
              const int o = slot & 1;
              pf[o] = st.x;
              pf[2 + o] = st.y;
              pf[4 + o] = st.z;
              pf[6 + o] = st.w;
            }
          }
          nt += __popc(km);
        }
        __syncwarp();
        if (WCUT) {
          // pairs for the packed loop; an odd tail is paired with a far-away
          // candidate of weight 0 (the clamp zeroes it)
          for (int h = lane; 2 * h < nt; h += 32) {
            const float4 c0 = sm.p[2 * h];
            const float4 c1 = 2 * h + 1 < nt ? sm.p[2 * h + 1] : make_float4(1e4f, 1e4f, 1e4f, 0.f);
            sm.pp[2 * h] = make_float4(c0.x, c1.x, c0.y, c1.y);
            sm.pp[2 * h + 1] = make_float4(c0.z, c1.z, c0.w, c1.w);
          }
        }
        if (PCOUNT) {
          for (int h = lane; 2 * h < nt; h += 32) {
            const float4 c0 = sm.p[2 * h];
            const float far = __int_as_float(0x7f800000);  // an odd tail: never counted
            const float4 c1 = 2 * h + 1 < nt ? sm.p[2 * h + 1] : make_float4(far, far, far, 0.f);
            sm.pp[2 * h] = make_float4(c0.x, c1.x, c0.y, c1.y);
            sm.pp[2 * h + 1] = make_float4(c0.z, c1.z, 0.f, 0.f);
          }
        }
        if (!WCUT && POL == POL_MATVEC && lane == 0 && (nt & 1)) {
          // pad an odd tile with a far-away candidate of weight 0 (finite, so
          // that every kernel formula stays finite and the clamp/select zeroes it)
          float *pf = reinterpret_cast<float *>(&sm.pp[2 * (nt >> 1)]);
          pf[1] = pf[3] = pf[5] = 1e4f;
          pf[7] = 0.f;
        }
        __syncwarp();
        float acc32 = 0.f;
        bool need = false;
        if (WCUT) {
          // one query against two candidates per packed FP32x2 instruction;
          // coordinates in units of the kernel support, so q = |dx|
          const float2 nqx = make_float2(-pq0 * sc, -pq0 * sc), nqy = make_float2(-pq1 * sc, -pq1 * sc),
                       nqz = make_float2(-pq2 * sc, -pq2 * sc);
          float2 acc2 = make_float2(0.f, 0.f);
          const int npair = (nt + 1) >> 1;
#pragma unroll 8
          for (int h = 0; h < npair; ++h) {
            const float4 A = sm.pp[2 * h], B = sm.pp[2 * h + 1];
            const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nqx);
            const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nqy);
            const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nqz);
            // d^2 (+1e-30, so that rsqrt stays finite for the self pair)
            float2 dd = __ffma2_rn(dx, dx, make_float2(1e-30f, 1e-30f));
            dd = __ffma2_rn(dy, dy, dd);
            dd = __ffma2_rn(dz, dz, dd);
            const float2 rs = make_float2(rsqrt_approx(dd.x), rsqrt_approx(dd.y));
            // t = max(1 - q, 0), q = d^2 / d, as saturating FMAs (q >= 0, so
            // [0,1] is the clamp); then 4q + 1 = 5 - 4t wherever t > 0
            const float2 t = make_float2(__saturatef(fmaf(-dd.x, rs.x, 1.f)),
                                         __saturatef(fmaf(-dd.y, rs.y, 1.f)));
            const float2 t2 = __fmul2_rn(t, t);
            const float2 pw = __ffma2_rn(t, make_float2(-4.f, -4.f), make_float2(5.f, 5.f));
            const float2 t4 = __fmul2_rn(t2, t2);
            acc2 = __ffma2_rn(__fmul2_rn(t4, pw), make_float2(B.z, B.w), acc2);
          }
          acc32 = acc2.x + acc2.y;
        } else if (POL == POL_MATVEC) {
          // one query against two candidates per packed FP32x2 instruction
          const float2 nqx = make_float2(-pq0, -pq0), nqy = make_float2(-pq1, -pq1),
                       nqz = make_float2(-pq2, -pq2);
          float2 acc2 = make_float2(0.f, 0.f);
          const int npair = (nt + 1) >> 1;
#pragma unroll 2
          for (int h = 0; h < npair; ++h) {
            const float4 A = sm.pp[2 * h], B = sm.pp[2 * h + 1];
            const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nqx);
            const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nqy);
            const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nqz);
            float2 dd = __fmul2_rn(dx, dx);
            dd = __ffma2_rn(dy, dy, dd);
            dd = __ffma2_rn(dz, dz, dd);
            // (a Wendland kernel here has a support wider than the radius: its value
            // does not vanish at the cut-off, see K_WEND_CUT)
            const bool ia = dd.x <= r2lo, ib = dd.y <= r2lo;
            need |= ((dd.x > r2lo) & (dd.x <= r2hi)) | ((dd.y > r2lo) & (dd.y <= r2hi));
            float2 w = kern32x2<KIND>(dd, P);
            w.x = ia ? w.x : 0.f;
            w.y = ib ? w.y : 0.f;
            acc2 = __ffma2_rn(w, make_float2(B.z, B.w), acc2);
          }
          acc32 = acc2.x + acc2.y;
        }
        if (PCOUNT) {
          // d^2 - mid for two candidates per packed instruction: the sign bit counts,
          // the smallest magnitude says whether any lies in the band
          const float2 nqx = make_float2(-pq0, -pq0), nqy = make_float2(-pq1, -pq1),
                       nqz = make_float2(-pq2, -pq2);
          const float2 nmid = make_float2(-r2mid, -r2mid);
          const int npair = (nt + 1) >> 1;
          float least = r2half + r2half;
          unsigned hits = 0;
#pragma unroll 8
          for (int h = 0; h < npair; ++h) {
            const float4 A = sm.pp[2 * h];
            const float2 B = *reinterpret_cast<const float2 *>(&sm.pp[2 * h + 1]);
            const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nqx);
            const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nqy);
            const float2 dz = __fadd2_rn(B, nqz);
            float2 dd = __fmul2_rn(dx, dx);
            dd = __ffma2_rn(dy, dy, dd);
            dd = __ffma2_rn(dz, dz, dd);
            const float2 off = __fadd2_rn(dd, nmid);
            hits += __float_as_uint(off.x) >> 31;
            hits += __float_as_uint(off.y) >> 31;
            least = fminf(least, fminf(fabsf(off.x), fabsf(off.y)));
          }
          count += (int)hits;
          need = least <= r2half;
        }
#pragma unroll 4
        for (int j = 0; j < nt && POL != POL_MATVEC && !PCOUNT; ++j) {
          const float4 c = sm.p[j];
          const float dd = norm32<NORM>(c.x - pq0, c.y - pq1, c.z - pq2);
          const bool in = dd <= r2lo;
          need |= (dd > r2lo) & (dd <= r2hi);
          if (POL == POL_COUNT) count += in ? 1 : 0;
          if (POL == POL_LIST && in && active) {
            const int2 mt = sm.meta[j];
            if (P.dx_out) write_dx(P, out_off, xq, mt.x, ws.seg[mt.y].z);
            P.cols_out[out_off++] = __float_as_int(c.w);
          }
        }
        if (!WCUT && __any_sync(0xffffffffu, need)) {
          // rare: decide the band pairs with the reference's FP64 test
          if (need) {
            if (!have_xq) {
              xq = P.qpos[qi];
              have_xq = true;
            }
            for (int j = 0; j < nt; ++j) {
              const float4 c = sm.p[j];
              const float dd = norm32<NORM>(c.x - pq0, c.y - pq1, c.z - pq2);
              const bool mid = PCOUNT && fabsf(__fadd_rn(dd, -r2mid)) <= r2half;
              const bool flagged = mid || (dd > r2lo && dd <= r2hi);
              if (flagged) {
                const int2 mt = sm.meta[j];
                int img[3], du0, du1;
                unpack_seg(ws.seg[mt.y].z, img, du0, du1);
                const bool inside = !(exact_norm(xq, P.cpos[mt.x], img, fg, NORM) > P.thr);
                if (PCOUNT) {
                  count += (inside ? 1 : 0) - (__fadd_rn(dd, -r2mid) < 0.f ? 1 : 0);
                } else if (inside) {
                  if (POL == POL_MATVEC) acc32 = fmaf(kern32<KIND>(dd, P), c.w, acc32);
                  if (POL == POL_COUNT) ++count;
                  if (POL == POL_LIST && active) {
                    if (P.dx_out) write_dx(P, out_off, xq, mt.x, ws.seg[mt.y].z);
                    P.cols_out[out_off++] = (int32_t)P.cperm[mt.x];
                  }
                }
              }
            }
          }
          __syncwarp();
        }
        if (POL == POL_MATVEC) acc64 += (double)acc32;
        __syncwarp();
      }
    }
    if (active) {
      if (POL == POL_MATVEC) P.c[P.qperm[qi]] = acc64;
      if (POL == POL_COUNT) P.counts_out[P.qperm[qi]] = count;
    }
  }
}

// Per-warp staging of the FP64 matvec: the candidates kept by the warp's
// bounding-box test, as FP32 offsets (for the prefilter) and as FP64
// positions shifted by their periodic image (x_j - image*L, for the kernel
// value), with their weights and (column index, segment) for the exact test.
// Two tiles in turn: a lane's neighbours left over from one are evaluated beside
// the next one's.
template <int KIND> struct WarpTile64 {
  // FP32 offsets as pairs of candidates: (x_a, x_b, y_a, y_b), (z_a, z_b)
  float4 pxy[STAGE / 2];
  float2 pz[STAGE / 2];
  // (bits of) the position: double, or fixed point (FIX)
  long long ux[2 * STAGE], uy[2 * STAGE], uz[2 * STAGE];
  double b[2 * STAGE], s[KIND == ABX_K_SCALAR_SUM ? 2 * STAGE : 1];
  // column and segment: of the last tile, of both where a value may want them
  static constexpr int METAS = KIND == ABX_K_LAPLACE ? 2 : 1;
  int2 meta[METAS * STAGE];
};

// FP64-accurate kernel value of one accepted pair from its fixed-point
// differences (fix64.cuh); the padding dimensions come first.
template <int KIND>
__device__ __forceinline__ double fix_value(long long dx, long long dy, long long dz,
                                            const KParams &P, const fx::u64 *tab, bool &near) {
  return fx::value<KIND>(dz, dy, dx, 3 - P.fg.eoff, P.fixc, tab, near);
}

// FP64 distance and kernel value of one accepted pair, dx = (x_j - image*L) - x_i; the
// image bits as in a segment (the centre one, whose shifts are 0, without them).
template <int KIND>
__device__ __forceinline__ double pair64(const D4 &xq, D4 xj, int code, const KParams &P, double si,
                                         double sj) {
  if ((code & 63) != CENTRE) {
    xj.x = __dsub_rn(xj.x, (double)((code & 3) - 1) * P.fg.L[0]);
    xj.y = __dsub_rn(xj.y, (double)(((code >> 2) & 3) - 1) * P.fg.L[1]);
    xj.z = __dsub_rn(xj.z, (double)(((code >> 4) & 3) - 1) * P.fg.L[2]);
  }
  const double dx = xj.x - xq.x, dy = xj.y - xq.y, dz = xj.z - xq.z;
  return kern64<KIND>(fma(dz, dz, fma(dy, dy, dx * dx)), P, si, sj);
}

// The same for a Laplace pair that the fixed-point value leaves out (k0 for a point
// with itself, or with one in the same place).
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ double near_pair64(const D4 &xq, int qi, int k, int code, const KParams &P) {
  const bool centre = (code & 63) == CENTRE;
  if (P.self && k == qi && centre) return P.fixc.k0;
  const D4 xj = P.cpos[k];
  if (centre && same_bits(xj.x, xq.x) && same_bits(xj.y, xq.y) && same_bits(xj.z, xq.z)) return P.fixc.k0;
  return pair64<ABX_K_LAPLACE>(xq, xj, code, P, 0.0, 0.0);
}

// FP64 sparse matvec: the reference's arithmetic for every accepted pair,
// FP64 work only for accepted pairs.  Per staged tile of <= 64 candidates:
//  (1) every lane classifies all candidates, two per packed FP32x2 instruction:
//      the sign of d2 - r2mid goes into a 64-bit mask of this lane's neighbours,
//      the least magnitude says whether any lies in the rounding band, where the
//      reference's exact FP64 test decides (rare);
//  (2) every lane walks its own mask and evaluates the FP64 distance, kernel
//      and product for those pairs only, until fewer than CARRY of the lanes
//      have any left; those are carried into the next tile's walk.
// A walk to the end of every tile costs the largest of 32 neighbour counts, of
// which 56 % of the lanes are busy on average (candidates of a tile lie
// together, the queries do not); two tiles at a time 74 %.  With FIX the values
// come from the integer units (fix64.cuh) and the FP64 pipe is left with one
// multiply-add a pair.  N = 1,048,576 clustered, 1,250 neighbours a row, Wendland:
// 103 -> 21.0 ms, with the packed test and the carried lanes 19.2 (issue slots 68 %
// busy, ALU 54 %, 21.7 lanes of 32).  The distance for the kernel value is |(x_j - image*L) - x_i|, which differs from the reference's
// x_j - (x_i + image*L) by at most an ulp of the box length (the acceptance
// decision itself is exact); the row sum order differs from the reference's.
constexpr int CARRY = 20;  // of 32 lanes: with fewer at work the rest of a tile waits for the next

template <int POL, int KIND, bool FIX>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32, 6)
    k_pairs_fp64(KParams P) {
  __shared__ WarpSeg seg_all[WARPS_PER_CTA];
  using Tile = WarpTile64<KIND>;
  __shared__ Tile tile_all[WARPS_PER_CTA];
  static_assert(POL == POL_MATVEC, "the FP64 pair kernel computes matvecs only");
  constexpr bool NEAR = FIX && KIND == ABX_K_LAPLACE;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpSeg &ws = seg_all[wid];
  Tile &sm = tile_all[wid];
  const FineGrid &fg = P.fg;
  const unsigned lt = (1u << lane) - 1u;
  const int nfull = P.counts[0], nunits = nfull + P.counts[P.all_units ? 1 : 8];
  if (blockIdx.x * WARPS_PER_CTA >= nunits) return;  // see grid_blocks
  __shared__ fx::u64 tab[FIX && KIND == ABX_K_GAUSSIAN ? fx::EXP_TAB : 1];
  if (FIX && KIND == ABX_K_GAUSSIAN) {
    for (int i = threadIdx.x; i < fx::EXP_TAB; i += WARPS_PER_CTA * 32) tab[i] = fx::exp_table.v[i];
    __syncthreads();
  }
  for (;;) {
    int unit = 0;
    if (lane == 0) unit = atomicAdd(P.counter, 1);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (unit >= nunits) break;
    const int2 U = unit < nfull ? P.units[unit] : P.units[P.units_cap - 1 - (unit - nfull)];
    const bool active = lane < U.y;
    const int qi = U.x + (active ? lane : 0);
    const int4 qc = P.qcell[qi];
    const float4 ql = P.qloc[qi];
    int lo[3], hi[3], a0, a1, R1, nrows;
    unit_box(P, qc, active, lo, hi, a0, a1, R1, nrows);
    const float pq0 = fmaf((float)(qc.x - lo[0]), fg.hf[0], ql.x);
    const float pq1 = fmaf((float)(qc.y - lo[1]), fg.hf[1], ql.y);
    const float pq2 = fmaf((float)(qc.z - lo[2]), fg.hf[2], ql.z);
    const float bl0 = warp_min(pq0), bh0 = warp_max(pq0);
    const float bl1 = warp_min(pq1), bh1 = warp_max(pq1);
    const float bl2 = warp_min(pq2), bh2 = warp_max(pq2);
    const float bc0 = 0.5f * (bl0 + bh0), bw0 = __fadd_ru(0.5f * (bh0 - bl0), 1e-6f * (fabsf(bl0) + fabsf(bh0)));
    const float bc1 = 0.5f * (bl1 + bh1), bw1 = __fadd_ru(0.5f * (bh1 - bl1), 1e-6f * (fabsf(bl1) + fabsf(bh1)));
    const float bc2 = 0.5f * (bl2 + bh2), bw2 = __fadd_ru(0.5f * (bh2 - bl2), 1e-6f * (fabsf(bl2) + fabsf(bh2)));
    // rounding band of the FP32 d2
    int span = 0;
#pragma unroll
    for (int e = 0; e < 3; ++e) span = max(span, hi[e] - lo[e] + 2 * fg.K[e] + 2);
    const TileBand bd = span < BAND_TAB ? TileBand{P.bands[2 * span], P.bands[2 * span + 1]}
                                        : tile_band(span, fg, P.r, P.r2, P.r2, 2);
    const float r2lo = bd.a.x, r2hi = bd.a.y, r2box = bd.a.z, r2mid = bd.b.x, r2half = bd.b.y;
    const D4 xq = P.qpos[qi];
    longlong2 fq = make_longlong2(0, 0);
    long long fqz = 0;
    if (FIX) {
      fq = P.qfxy[qi];
      fq = make_longlong2(fx::biased(fq.x), fx::biased(fq.y));
      fqz = fx::biased(P.qfz[qi]);
    }
    const double si = (KIND == ABX_K_SCALAR_SUM) ? P.s_row[qi] : 0.0;
    double acc = 0.0;
    const int few = U.y * CARRY / 32;
    unsigned long long left = 0;  // this lane's neighbours in the tile before
    int half = 0;                 // 0 or STAGE: the slots of the tile being staged
    auto evaluate = [&](int j) {  // distance, kernel and product of the pair in slot j
      double v;
      if (FIX) {
        bool near;
        v = fix_value<KIND>(fx::diff(sm.ux[j], fq.x), fx::diff(sm.uy[j], fq.y),
                            fx::diff(sm.uz[j], fqz), P, tab, near);
        if (NEAR && near) {
          const int2 mt = sm.meta[j & (Tile::METAS * STAGE - 1)];
          v = near_pair64(xq, qi, mt.x, mt.y, P);
        }
      } else {
        const double dx = __longlong_as_double(sm.ux[j]) - xq.x,
                     dy = __longlong_as_double(sm.uy[j]) - xq.y,
                     dz = __longlong_as_double(sm.uz[j]) - xq.z;
        v = kern64<KIND>(fma(dz, dz, fma(dy, dy, dx * dx)), P, si,
                         KIND == ABX_K_SCALAR_SUM ? sm.s[j] : 0.0);
      }
      acc = fma(v, sm.b[j], acc);
    };

    for (int row0 = 0; row0 < nrows; row0 += 32) {
      const int nseg = build_segments(P, lo, hi, a0, a1, R1, nrows, row0, ws, lane);
      if (nseg == 0) continue;
      const int total = ws.off[nseg];
      int cur = 0;
      for (int t0 = 0; t0 < total; t0 += STAGE) {
        constexpr int NS = STAGE / 32;
        int kk[NS], sx[NS];
        float4 so[NS];
#pragma unroll
        for (int sub = 0; sub < NS; ++sub) {
          const int t = t0 + sub * 32 + lane;
          kk[sub] = -1;
          sx[sub] = 0;
          so[sub] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (t < total) {
            while (cur + 1 < nseg && ws.off[cur + 1] <= t) ++cur;
            sx[sub] = cur;
            kk[sub] = ws.seg[cur].x + (t - ws.off[cur]);
            so[sub] = ws.segf[cur];
          }
        }
        float4 cls[NS];
#pragma unroll
        for (int sub = 0; sub < NS; ++sub)
          cls[sub] = kk[sub] >= 0 ? __ldg(&P.cloc[kk[sub]]) : make_float4(0.f, 0.f, 0.f, 0.f);
        int nt = 0;
#pragma unroll
        for (int sub = 0; sub < NS; ++sub) {
          bool keep = false;
          float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
          const int k = kk[sub];
          if (k >= 0) {
            const float4 cl = cls[sub];
            st.x = fmaf(so[sub].x, fg.hf[0], cl.x);
            st.y = fmaf(so[sub].y, fg.hf[1], cl.y);
            st.z = fmaf(cl.w + so[sub].z, fg.hf[2], cl.z);
            const float e0 = fmaxf(fabsf(st.x - bc0) - bw0, 0.f);
            const float e1 = fmaxf(fabsf(st.y - bc1) - bw1, 0.f);
            const float e2 = fmaxf(fabsf(st.z - bc2) - bw2, 0.f);
            keep = fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) <= r2box;
          }
          const unsigned km = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            const int slot = nt + __popc(km & lt);
            int img[3], du0, du1;
            unpack_seg(ws.seg[sx[sub]].z, img, du0, du1);
            float *xy = reinterpret_cast<float *>(&sm.pxy[slot >> 1]) + (slot & 1);
            xy[0] = st.x;
            xy[2] = st.y;
            reinterpret_cast<float *>(sm.pz)[slot] = st.z;
            const int at = half + slot;
            if (FIX) {
              const longlong2 f = P.fxy[k];
              sm.ux[at] = fx::diff(f.x, img[0] * P.Lfix[0]);
              sm.uy[at] = fx::diff(f.y, img[1] * P.Lfix[1]);
              sm.uz[at] = fx::diff(P.fz[k], img[2] * P.Lfix[2]);
            } else {
              const D4 pj = P.cpos[k];
              sm.ux[at] = __double_as_longlong(__dsub_rn(pj.x, (double)img[0] * fg.L[0]));
              sm.uy[at] = __double_as_longlong(__dsub_rn(pj.y, (double)img[1] * fg.L[1]));
              sm.uz[at] = __double_as_longlong(__dsub_rn(pj.z, (double)img[2] * fg.L[2]));
            }
            sm.b[at] = P.b64[k];
            if (KIND == ABX_K_SCALAR_SUM) sm.s[at] = P.s_col[k];
            sm.meta[at & (Tile::METAS * STAGE - 1)] = make_int2(k, ws.seg[sx[sub]].z);
          }
          nt += __popc(km);
        }
        if (nt == 0) continue;  // (in 1-D most tiles lie beyond the unit's reach)
        __syncwarp();
        if (lane == 0 && (nt & 1)) {  // an odd tail is paired with a candidate at infinity
          float *xy = reinterpret_cast<float *>(&sm.pxy[nt >> 1]);
          xy[1] = xy[3] = __int_as_float(0x7f800000);
          reinterpret_cast<float *>(sm.pz)[nt] = __int_as_float(0x7f800000);
        }
        __syncwarp();
        // (1) this lane's neighbours among the nt staged candidates
        unsigned long long mask = 0, nmask = 0;  // nmask: those that go by FP64
        if (active) {
          const float2 nqx = make_float2(-pq0, -pq0), nqy = make_float2(-pq1, -pq1),
                       nqz = make_float2(-pq2, -pq2), nmid = make_float2(-r2mid, -r2mid);
          const float2 nnear = make_float2(r2mid - P.near2, r2mid - P.near2);
          float least = r2half + r2half;
          unsigned word[2] = {0u, 0u}, nword[2] = {0u, 0u};
          const int npair = (nt + 1) >> 1;
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int n16 = min(max(npair - 16 * w, 0), 16);
#pragma unroll 4
            for (int h = 0; h < n16; ++h) {
              const float4 A = sm.pxy[16 * w + h];
              const float2 B = sm.pz[16 * w + h];
              const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nqx);
              const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nqy);
              const float2 dz = __fadd2_rn(B, nqz);
              float2 dd = __fmul2_rn(dx, dx);
              dd = __ffma2_rn(dy, dy, dd);
              dd = __ffma2_rn(dz, dz, dd);
              const float2 off = __fadd2_rn(dd, nmid);
              word[w] = __funnelshift_l(__float_as_uint(off.x), word[w], 1);
              word[w] = __funnelshift_l(__float_as_uint(off.y), word[w], 1);
              least = fminf(least, fminf(fabsf(off.x), fabsf(off.y)));
              if (NEAR) {
                const float2 no = __fadd2_rn(off, nnear);  // d^2 - near2
                nword[w] = __funnelshift_l(__float_as_uint(no.x), nword[w], 1);
                nword[w] = __funnelshift_l(__float_as_uint(no.y), nword[w], 1);
              }
            }
            // the first candidate's sign to bit 0
            if (n16) word[w] = __brev(word[w] << (32 - 2 * n16));
            if (NEAR && n16) nword[w] = __brev(nword[w] << (32 - 2 * n16));
          }
          mask = word[0] | (unsigned long long)word[1] << 32;
          if (NEAR) nmask = nword[0] | (unsigned long long)nword[1] << 32;
          if (least <= r2half) {  // rare: the reference's exact FP64 test for pairs in the band
            for (int j = 0; j < nt; ++j) {
              const float *xy = reinterpret_cast<const float *>(&sm.pxy[j >> 1]) + (j & 1);
              const float d0 = xy[0] - pq0, d1 = xy[2] - pq1,
                          d2v = reinterpret_cast<const float *>(sm.pz)[j] - pq2;
              const float dd = fmaf(d2v, d2v, fmaf(d1, d1, d0 * d0));
              if (!(fabsf(dd - r2mid) <= r2half) && !(dd > r2lo && dd <= r2hi)) continue;
              const int2 mt = sm.meta[(half + j) & (Tile::METAS * STAGE - 1)];
              int img[3], du0, du1;
              unpack_seg(mt.y, img, du0, du1);
              const bool in = !(exact_d2(xq, P.cpos[mt.x], img, fg) > P.r2);
              mask = in ? mask | 1ull << j : mask & ~(1ull << j);
            }
          }
        }
        if (NEAR) {  // together, so that a clump of near pairs is not a walk of both kinds
          nmask &= mask;
          mask &= ~nmask;
          while (__any_sync(0xffffffffu, nmask != 0)) {
            if (nmask != 0) {
              const int j = half + __ffsll((long long)nmask) - 1;
              nmask &= nmask - 1;
              const int2 mt = sm.meta[j];
              acc = fma(near_pair64(xq, qi, mt.x, mt.y, P), sm.b[j], acc);
            }
          }
        }
        // (2) what is left of the tile before, together with this one's
        while (__any_sync(0xffffffffu, left != 0)) {
          const bool old = left != 0;
          unsigned long long &from = old ? left : mask;
          if (from != 0) {
            const int j = __ffsll((long long)from) - 1;
            from &= from - 1;
            evaluate((old ? half ^ STAGE : half) + j);
          }
        }
        while (__popc(__ballot_sync(0xffffffffu, mask != 0)) > few) {
          if (mask != 0) {
            const int j = __ffsll((long long)mask) - 1;
            mask &= mask - 1;
            evaluate(half + j);
          }
        }
        left = mask;
        half ^= STAGE;
        __syncwarp();
      }
    }
    while (__any_sync(0xffffffffu, left != 0)) {
      if (left != 0) {
        const int j = __ffsll((long long)left) - 1;
        left &= left - 1;
        evaluate((half ^ STAGE) + j);
      }
    }
    __syncwarp();
    if (active) P.c[P.qperm[qi]] = acc;
  }
}

// ----------------------------------------------- few lanes a query ---
// The pair work of the small units (few queries in GROUP_E2 cells: up to ~150
// neighbours a ball in 3-D), where a warp of the unit kernels would keep most
// lanes idle.  A query has P.lanes lanes (a power of two), which share the rows
// of its stencil: one where there are queries enough to fill the GPU, up to a
// whole warp for small sets, whose time is the latency of one query's rows.
// The FP32 test is as cheap as the loads; FP64 values (~100 instructions) are
// not evaluated where they are found but queued per lane in shared memory and
// evaluated when a queue is full, as long as DRAIN lanes have one.  N = 100,000,
// 50 neighbours a row: a count of 100,000 moved points 2,060 -> 474 us (330 with
// the sorts of primitives.cu), FP64 Gaussian product 3,229 -> 197 us.
enum { VAL_FP64 = 0, VAL_MIXED = 1, VAL_FIX = 2 };
constexpr int QCAP = 16;   // queued pairs per lane
constexpr int DRAIN = 22;  // lanes that make an evaluation worth its issue
constexpr uint32_t FLUSH32 = 32;  // terms from which on an FP32 sum goes to the FP64 one (below twice that)

template <int POL, int KIND, int VAL, int NORM = 2>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32)
    k_pairs_thread(KParams P) {
  constexpr bool QUEUE = POL == POL_MATVEC && VAL != VAL_MIXED;
  constexpr bool WCUT = KIND == K_WEND_CUT;
  constexpr bool NEAR = VAL == VAL_FIX && KIND == ABX_K_LAPLACE;
  constexpr int NEAR_CODE = 64;  // beside the image bits of a queued pair
  __shared__ unsigned long long queue[QUEUE ? WARPS_PER_CTA * QCAP * 32 : 1];
  __shared__ fx::u64 tab[VAL == VAL_FIX && KIND == ABX_K_GAUSSIAN ? fx::EXP_TAB : 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long *qu = queue + (QUEUE ? wid * QCAP * 32 + lane : 0);
  const FineGrid &fg = P.fg;
  if (VAL == VAL_FIX && KIND == ABX_K_GAUSSIAN) {
    for (int i = threadIdx.x; i < fx::EXP_TAB; i += WARPS_PER_CTA * 32) tab[i] = fx::exp_table.v[i];
    __syncthreads();
  }
  const int nsing = P.counts[9], nrows = P.counts[3];
  if ((int64_t)blockIdx.x * (WARPS_PER_CTA * 32) >= (int64_t)nsing * P.lanes) return;  // see grid_blocks
  const int sub = lane & (P.lanes - 1);
  const int span = 2 * max(max(fg.K[0], fg.K[1]), fg.K[2]) + 2;
  const float4 bd = span < BAND_TAB ? P.bands[2 * span]
                                    : tile_band(span, fg, P.r, P.r2, P.thr, NORM).a;
  const float r2lo = bd.x, r2hi = bd.y;
  const float p0f2 = WCUT ? P.p0f * P.p0f : 0.f;
  for (;;) {
    int base = 0;
    if (lane == 0) base = atomicAdd(P.counter + 1, 32 / P.lanes);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= nsing) break;
    const int mine = base + lane / P.lanes;
    const bool act = mine < nsing;
    const int qi = P.singles[act ? mine : base];
    const int4 qc = P.qcell[qi];
    const float4 ql = P.qloc[qi];
    D4 xq;
    if (QUEUE && VAL == VAL_FP64) xq = P.qpos[qi];
    longlong2 fq = make_longlong2(0, 0);
    long long fqz = 0;
    if (VAL == VAL_FIX) {
      fq = P.qfxy[qi];
      fq = make_longlong2(fx::biased(fq.x), fx::biased(fq.y));
      fqz = fx::biased(P.qfz[qi]);
    }
    const double si = (QUEUE && KIND == ABX_K_SCALAR_SUM) ? P.s_row[qi] : 0.0;
    double acc = 0.0;
    float acc32 = 0.f;
    int count = 0, nq = 0;
    uint32_t terms = 0;  // candidates since this lane's FP32 sum was handed on
    auto evaluate = [&]() {  // one queued pair of every lane that has one
      if (nq > 0) {
        --nq;
        const unsigned long long ent = qu[nq * 32];
        const unsigned k = (unsigned)ent;
        const int code = (int)(ent >> 32);
        double v;
        if (NEAR && (code & NEAR_CODE)) {
          v = near_pair64(P.qpos[qi], qi, (int)k, code, P);
        } else if (VAL == VAL_FIX) {
          const longlong2 f = P.fxy[k];
          long long dx = fx::diff(f.x, fq.x), dy = fx::diff(f.y, fq.y), dz = fx::diff(P.fz[k], fqz);
          if (code != CENTRE) {
            dx = fx::diff(dx, ((code & 3) - 1) * P.Lfix[0]);
            dy = fx::diff(dy, (((code >> 2) & 3) - 1) * P.Lfix[1]);
            dz = fx::diff(dz, (((code >> 4) & 3) - 1) * P.Lfix[2]);
          }
          bool near;
          v = fix_value<KIND>(dx, dy, dz, P, tab, near);
          if (NEAR && near) v = near_pair64(P.qpos[qi], qi, (int)k, code, P);
        } else
          v = pair64<KIND>(xq, P.cpos[k], code, P, si, KIND == ABX_K_SCALAR_SUM ? P.s_col[k] : 0.0);
        acc = fma(v, P.b64[k], acc);
      }
    };
    for (int t0 = 0; t0 < nrows; t0 += P.lanes) {
      const bool has = t0 + sub < nrows;
      const int4 st = P.stencil[has ? t0 + sub : 0];  // o0, o1, reach along e2
      {
        int w0 = qc.x + st.x, i0 = 1, w1 = qc.y + st.y, i1 = 1;
        bool ok = act && has;
        if (w0 < 0) {
          ok = ok && fg.periodic[0] && w0 >= -fg.m[0];
          w0 += fg.m[0];
          i0 = 2;
        } else if (w0 >= fg.m[0]) {
          ok = ok && fg.periodic[0] && w0 < 2 * fg.m[0];
          w0 -= fg.m[0];
          i0 = 0;
        }
        if (w1 < 0) {
          ok = ok && fg.periodic[1] && w1 >= -fg.m[1];
          w1 += fg.m[1];
          i1 = 2;
        } else if (w1 >= fg.m[1]) {
          ok = ok && fg.periodic[1] && w1 < 2 * fg.m[1];
          w1 -= fg.m[1];
          i1 = 0;
        }
        const int a2 = qc.z - st.z, b2 = qc.z + st.z;
        const int m2 = fg.m[2];
        const uint32_t row = ok ? ((uint32_t)w0 * fg.m[1] + w1) * (uint32_t)m2 : 0u;
        const float rx = fmaf((float)st.x, fg.hf[0], -ql.x), ry = fmaf((float)st.y, fg.hf[1], -ql.y);
        // the domain itself, then (periodic e2) its images below and above
        for (int part = 0; part < 3; ++part) {
          const int i2 = part == 0 ? 0 : (part == 1 ? 1 : -1);  // image; wrapped w2 = u2 + i2 m2
          const int sa = max(a2 + i2 * m2, 0), sb = min(b2 + i2 * m2, m2 - 1);
          const bool some = ok && sa <= sb;
          if (part > 0) {
            if (!fg.periodic[2]) break;
            if (!__any_sync(0xffffffffu, some)) continue;
          }
          uint32_t k = 0, e = 0;
          if (some) {
            k = P.cell_start[row + (uint32_t)sa];
            e = P.cell_start[row + (uint32_t)sb + 1];
          }
          const float zs = (float)(-i2 * m2 - qc.z);
          const int code = i0 | (i1 << 2) | ((i2 + 1) << 4);
          // mixed sums: at most FLUSH32 candidates of a row at a time, which may cross a
          // cluster that the query is not in
          constexpr bool SUM32 = VAL == VAL_MIXED && POL == POL_MATVEC;
          for (;;) {
            const uint32_t to = SUM32 ? min(e, k + FLUSH32) : e;
            if (SUM32) terms += to - k;
            while (__any_sync(0xffffffffu, k < to)) {
              if (k < to) {
                const float4 cl = __ldg(&P.cloc[k]);
                const float dx = cl.x + rx, dy = cl.y + ry,
                            dz = fmaf(cl.w + zs, fg.hf[2], cl.z) - ql.z;
                float dd = norm32<NORM>(dx, dy, dz);
                if (WCUT) {
                  // the clamp is the cut-off (see K_WEND_CUT)
                  dd = fmaf(dd, p0f2, 1e-30f);
                  const float t = __saturatef(fmaf(-dd, rsqrt_approx(dd), 1.f));
                  const float t2 = t * t;
                  if (t > 0.f) acc32 = fmaf(t2 * t2 * fmaf(t, -4.f, 5.f), __ldg(&P.b32[k]), acc32);
                } else {
                  bool in = dd <= r2lo;
                  if (!in && dd <= r2hi) {  // rare: the reference's FP64 test
                    // (opaque: otherwise the image shifts' FP64 products are computed for
                    // every row, ahead of this branch; 100,000 x 50 Gaussian 197 -> 192 us)
                    int img[3] = {i0 - 1, i1 - 1, i2};
                    asm volatile("" : "+r"(img[0]), "+r"(img[1]), "+r"(img[2]));
                    in = !(exact_norm(P.qpos[qi], P.cpos[k], img, fg, NORM) > P.thr);
                  }
                  if (POL == POL_COUNT) count += in ? 1 : 0;
                  if (POL == POL_MATVEC && VAL == VAL_MIXED && in)
                    acc32 = fmaf(kern32<KIND>(dd, P), __ldg(&P.b32[k]), acc32);
                  if (QUEUE && in) {
                    const int c = NEAR && dd < P.near2 ? code | NEAR_CODE : code;
                    qu[nq * 32] = (unsigned long long)k | ((unsigned long long)c << 32);
                    ++nq;
                  }
                }
                ++k;
              }
              if (QUEUE && __any_sync(0xffffffffu, nq == QCAP)) {
                do evaluate();
                while (__popc(__ballot_sync(0xffffffffu, nq > 0)) >= DRAIN);
              }
            }
            if (!SUM32 || !__any_sync(0xffffffffu, terms >= FLUSH32)) break;
            acc += (double)acc32;
            acc32 = 0.f;
            terms = 0;
            if (!__any_sync(0xffffffffu, k < e)) break;
          }
        }
      }
    }
    if (QUEUE)
      while (__any_sync(0xffffffffu, nq > 0)) evaluate();
    if (POL == POL_MATVEC && VAL == VAL_MIXED) acc += (double)acc32;
    for (int d = 1; d < P.lanes; d <<= 1) {
      if (POL == POL_MATVEC) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (POL == POL_COUNT) count += __shfl_xor_sync(0xffffffffu, count, d);
    }
    if (act && sub == 0) {
      if (POL == POL_MATVEC) P.c[P.qperm[qi]] = acc;
      if (POL == POL_COUNT) P.counts_out[P.qperm[qi]] = count;
    }
  }
}

// b in the columns' kernel order; zeroes the pair kernels' work counters.
__global__ void k_gather_b(const double *__restrict__ b, const uint32_t *__restrict__ perm,
                           int64_t n, float *__restrict__ b32, double *__restrict__ b64,
                           int *__restrict__ counters) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0 && counters) counters[0] = counters[1] = 0;
  if (k >= n) return;
  const double v = b[perm[k]];
  if (b32) b32[k] = (float)v;
  if (b64) b64[k] = v;
}

double prune_distance2(const PairLayout &L) {
  double hmax = 0;
  for (int e = 0; e < 3; ++e)
    if (e >= L.fg.eoff) hmax = std::max(hmax, L.fg.h[e]);
  const double margin = L.r * 1e-9 + hmax * 1e-9;
  return (L.r + margin) * (L.r + margin);
}

int build_tables(abx_context *ctx, PairLayout &L, int norm, double thr) {
  ABX_TRY(L.ext.reserve(EXT_TAB * EXT_TAB));
  ABX_TRY(L.bands.reserve(2 * BAND_TAB));
  ABX_TRY(L.stencil.reserve(ROWS_MAX));
  k_tables<<<EXT_TAB * EXT_TAB / TABLE_TPB, TABLE_TPB, 0, ctx->stream>>>(
      L.fg, prune_distance2(L), L.r, thr, norm, L.ext.ptr, L.bands.ptr, L.stencil.ptr,
      L.counts.ptr, (int)L.rows->n, L.split.fold, L.work, ++L.work_seq);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

// The units anew for another split, in the same buffers.
int relist_units(abx_context *ctx, PairLayout &L, const Split &split) {
  ABX_TRY(build_units(ctx, L, split));
  return build_tables(ctx, L, 2, L.r * L.r);
}

KParams base_params(const PairLayout &L) {
  KParams P{};
  P.ext = L.ext.ptr;
  P.bands = L.bands.ptr;
  P.stencil = L.stencil.ptr;
  P.fg = L.fg;
  P.r = L.r;
  P.r2 = L.r * L.r;
  P.lnorm = 2;
  P.thr = P.r2;
  P.prune2 = prune_distance2(L);
  P.cloc = L.cols.loc.ptr;
  P.cpos = L.cols.posk.ptr;
  P.cell_start = L.cell_start.ptr;
  P.cperm = L.cols.perm.ptr;
  P.qcell = L.rows->cell.ptr;
  P.qloc = L.rows->loc.ptr;
  P.qpos = L.rows->posk.ptr;
  P.units = L.units.ptr;
  P.units_cap = L.rows->n;
  P.singles = L.singles.ptr;
  P.counts = L.counts.ptr;
  P.counter = L.counts.ptr + 4;
  P.qperm = L.rows->perm.ptr;
  P.self = L.self;
  // R / 128 (fx::laplace_far), with room for the FP32 distances: the value itself
  // says what is left out
  P.near2 = (float)std::ldexp(1.0 + 1e-3, 2 * (L.unit.r - 7));
  P.work = L.work ? unit_work(L.work, L.work_seq) : UnitWork{true, true};
  P.fxy = L.cols.fxy.ptr;
  P.fz = L.cols.fz.ptr;
  P.qfxy = L.rows->fxy.ptr;
  P.qfz = L.rows->fz.ptr;
  if (L.unit.ok)
    for (int e = 0; e < 3; ++e) P.Lfix[e] = fx::to_fixed(L.fg.L[e], L.unit.f, L.unit.k);
  return P;
}

// CTAs of the kernels that take their work from a counter: as many as there
// can be work for, 8 an SM at most.  How much there is only the device knows; CTAs
// beyond it return at once, as the first ones, which are dealt evenly over the SMs,
// would not get it all otherwise (300 clumps of 200 points, whose 2,200 units would
// fill a quarter of the warps: busiest SM 1.69e6 cycles, 1.25e6 with as many CTAs as
// units; average 1.03e6).
int grid_blocks(abx_context *ctx, const KParams &P) {
  const int64_t need = (P.units_cap + WARPS_PER_CTA - 1) / WARPS_PER_CTA;
  return (int)std::max<int64_t>(1, std::min<int64_t>(ctx->num_sms * 8, need));
}
// Lanes a query of the singles: enough queries x lanes for LANES_FILL an SM.
constexpr int64_t LANES_FILL = 2048;
int query_lanes(abx_context *ctx, int64_t nq) {
  int g = 1;
  while (g < 32 && nq * g < ctx->num_sms * LANES_FILL) g *= 2;
  return g;
}
int thread_blocks(abx_context *ctx, const KParams &P) {
  const int64_t need = (P.units_cap * P.lanes + WARPS_PER_CTA * 32 - 1) / (WARPS_PER_CTA * 32);
  return (int)std::max<int64_t>(1, std::min<int64_t>(ctx->num_sms * 12, need));
}
// The full units by a warp each, the small units' queries by P.lanes lanes each.
template <int KIND> int launch_matvec(abx_context *ctx, KParams P, bool mixed, bool fix) {
  cudaStream_t s = ctx->stream;
  P.lanes = query_lanes(ctx, P.units_cap);
  const int ub = grid_blocks(ctx, P), tb = thread_blocks(ctx, P), T = WARPS_PER_CTA * 32;
  // the two Gaussians are one kernel where it matters
  constexpr int FK = KIND == ABX_K_COMPACT_GAUSSIAN ? ABX_K_GAUSSIAN : KIND;
  constexpr bool CAN_FIX = FK == ABX_K_GAUSSIAN || FK == ABX_K_WENDLAND_C2 ||
                           FK == ABX_K_LAPLACE || FK == ABX_K_MULTIQUADRIC;
  const bool units = P.work.full, singles = P.work.singles;
  if (mixed) {
    if (units) k_pairs_mixed<POL_MATVEC, FK><<<ub, T, 0, s>>>(P);
    if (singles) k_pairs_thread<POL_MATVEC, FK, VAL_MIXED><<<tb, T, 0, s>>>(P);
  } else {
    if constexpr (CAN_FIX) {
      if (fix) {
        if (units) k_pairs_fp64<POL_MATVEC, FK, true><<<ub, T, 0, s>>>(P);
        if (singles) k_pairs_thread<POL_MATVEC, FK, VAL_FIX><<<tb, T, 0, s>>>(P);
        ABX_CHECK_CUDA(cudaGetLastError());
        return ABX_OK;
      }
    }
    if constexpr (KIND != K_WEND_CUT) {
      if (units) k_pairs_fp64<POL_MATVEC, FK, false><<<ub, T, 0, s>>>(P);
      if (singles) k_pairs_thread<POL_MATVEC, FK, VAL_FP64><<<tb, T, 0, s>>>(P);
    }
  }
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

// The radius search (count or list) in the norm P.lnorm.  Lists keep one
// kernel for all units: their order within a row is the unit kernel's.
template <int POL, int NORM> int launch_search_norm(abx_context *ctx, KParams P) {
  cudaStream_t s = ctx->stream;
  const int T = WARPS_PER_CTA * 32;
  P.all_units = POL == POL_LIST ? 1 : 0;
  P.lanes = query_lanes(ctx, P.units_cap);
  if (POL == POL_LIST) P.counter += 2;  // (zeroed by the layout, as the count's are)
  k_pairs_mixed<POL, ABX_K_CONST, NORM><<<grid_blocks(ctx, P), T, 0, s>>>(P);
  if (POL == POL_COUNT)
    k_pairs_thread<POL_COUNT, ABX_K_CONST, VAL_MIXED, NORM><<<thread_blocks(ctx, P), T, 0, s>>>(P);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}
template <int POL> int launch_search(abx_context *ctx, const KParams &P) {
  if (P.lnorm == 1) return launch_search_norm<POL, 1>(ctx, P);
  if (P.lnorm == -1) return launch_search_norm<POL, -1>(ctx, P);
  return launch_search_norm<POL, 2>(ctx, P);
}

int launch_matvec_kind(abx_context *ctx, const KParams &P, bool mixed, bool fix) {
  switch (P.kind) {
  case ABX_K_CONST: return launch_matvec<ABX_K_CONST>(ctx, P, mixed, fix);
  case ABX_K_GAUSSIAN:
  case ABX_K_COMPACT_GAUSSIAN: return launch_matvec<ABX_K_GAUSSIAN>(ctx, P, mixed, fix);
  case ABX_K_WENDLAND_C2:
    // support 1/p0 <= r up to rounding of p0 = 1/r (a support wider by a
    // relative 1e-9 adds pairs of weight <= 5e-36)
    if (mixed && P.p0 * P.r >= 1.0 - 1e-9) return launch_matvec<K_WEND_CUT>(ctx, P, true, false);
    return launch_matvec<ABX_K_WENDLAND_C2>(ctx, P, mixed, fix);
  case ABX_K_LAPLACE: return launch_matvec<ABX_K_LAPLACE>(ctx, P, mixed, fix);
  case ABX_K_MULTIQUADRIC: return launch_matvec<ABX_K_MULTIQUADRIC>(ctx, P, mixed, fix);
  case ABX_K_SCALAR_SUM: return launch_matvec<ABX_K_SCALAR_SUM>(ctx, P, false, false);
  }
  set_error("unknown kernel kind %d", P.kind);
  return ABX_ERR_INVALID;
}

int fill_fixed(abx_context *ctx, PointLayout &P, const fx::Unit &U) {
  ABX_TRY(P.fxy.reserve(P.n ? P.n : 1));
  ABX_TRY(P.fz.reserve(P.n ? P.n : 1));
  if (P.n)
    k_fill_fixed<<<ceil_div(P.n, TPB), TPB, 0, ctx->stream>>>(P.posk.ptr, P.n, U, P.fxy.ptr,
                                                              P.fz.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

// Build a layout for cols (a searchable particle set) and a query set given as
// SoA FP64 (qsrc, nq, stride) -- or the column set itself when qsrc == null.
// All on the context's stream, nothing waited for; norm and thr as KParams'; units
// false: the points and cells alone.
int layout_build(abx_context *ctx, abx_particles *cols, double r, const double *qsrc, int64_t nq,
                 int64_t qstride, PairLayout &L, const Split &split, int norm = 2,
                 bool units = true) {
  GridDesc g;
  ABX_TRY(particles_grid_desc(cols, &g));
  L.r = r;
  L.fg = make_fine_grid(g, r, std::max<int64_t>(cols->n, 1), 3);
  PointSets sets{};
  ABX_TRY(reserve_points(cols->n, cols->pos.ptr, cols->n, true, L.cols, sets.s[0]));
  L.self = !qsrc;
  L.rows = L.self ? &L.cols : &L.rows_own;
  if (!L.self) ABX_TRY(reserve_points(nq, qsrc, qstride, false, L.rows_own, sets.s[1]));
  ABX_TRY(build_points(ctx, sets, L.cols, L.self ? nullptr : &L.rows_own, L.fg));
  ABX_TRY(build_cell_start(ctx, L));
  if (!units) return ABX_OK;
  ABX_TRY(build_units(ctx, L, split));
  ABX_TRY(build_tables(ctx, L, norm, norm == 2 ? r * r : std::fabs(r)));
  return ABX_OK;
}

}  // namespace

// The unit of an operator's FP64 product on the integer units (fix64.cuh).
fx::Unit fix_unit(const abx_kernel &k, double reach) {
  switch (k.kind) {
  case ABX_K_GAUSSIAN:
  case ABX_K_COMPACT_GAUSSIAN: return fx::make_unit<fx::GAUSSIAN>(k.p[0], reach);
  case ABX_K_WENDLAND_C2: return fx::make_unit<fx::WENDLAND>(k.p[0], reach);
  case ABX_K_LAPLACE: return fx::make_unit<fx::LAPLACE>(k.p[0], reach);
  case ABX_K_MULTIQUADRIC: return fx::make_unit<fx::MULTIQUADRIC>(k.p[0], reach);
  default: return fx::Unit{};
  }
}

static Split matvec_split(const abx_operator *op) {
  if (op->precision == ABX_PREC_MIXED && op->k.kind != ABX_K_SCALAR_SUM)
    return op->rows->n < MIXED_MIN ? SPLIT_NONE : SPLIT_MIXED;
  if (op->cols->dim == 1) return SPLIT_NONE;
  return fix_unit(op->k, op->radius).ok ? SPLIT_FP64 : SPLIT_VALUES;
}

int pair_layout_build(abx_operator *op) {
  abx_context *ctx = op->rows->ctx;
  if (!op->pairs) op->pairs = new PairLayout();
  PairLayout &L = *op->pairs;  // a rebuild keeps the buffers
  if (!L.work) {
    ABX_CHECK_CUDA(cudaHostAlloc((void **)&L.work, sizeof(uint64_t), cudaHostAllocMapped));
    *L.work = 0;
  }
  L.cols_version = ~uint64_t(0);  // valid once everything below has succeeded
  const bool self = op->rows == op->cols;
  ABX_TRY(layout_build(ctx, op->cols, op->radius, self ? nullptr : op->rows->pos.ptr,
                       op->rows->n, op->rows->n, L, matvec_split(op)));
  L.rows_version = op->rows->version;
  L.unit = fix_unit(op->k, L.r);
  if (L.unit.ok) {
    ABX_TRY(fill_fixed(ctx, L.cols, L.unit));
    if (!L.self) ABX_TRY(fill_fixed(ctx, L.rows_own, L.unit));
  }
  const int64_t nr = L.rows->n, nc = L.cols.n;
  ABX_TRY(L.bk32.reserve(nc ? nc : 1));
  ABX_TRY(L.bk64.reserve(nc ? nc : 1));
  if (op->k.kind == ABX_K_SCALAR_SUM) {
    ABX_REQUIRE(op->rows->has_scalar && op->cols->has_scalar, ABX_ERR_STATE,
                "ABX_K_SCALAR_SUM needs a scalar column on both particle sets");
    ABX_TRY(L.sk.reserve(nc ? nc : 1));
    ABX_TRY(L.sq.reserve(nr ? nr : 1));
    if (nc)
      k_gather_b<<<ceil_div(nc, TPB), TPB, 0, ctx->stream>>>(op->cols->scalar.ptr, L.cols.perm.ptr,
                                                             nc, nullptr, L.sk.ptr, nullptr);
    if (nr)
      k_gather_b<<<ceil_div(nr, TPB), TPB, 0, ctx->stream>>>(op->rows->scalar.ptr, L.rows->perm.ptr,
                                                             nr, nullptr, L.sq.ptr, nullptr);
    ABX_CHECK_CUDA(cudaGetLastError());
  }
  L.cols_version = op->cols->version;
  return ABX_OK;
}

int sparse_matvec_device(abx_operator *op, const double *b, double *c) {
  abx_context *ctx = op->rows->ctx;
  if (!op->pairs || op->pairs->cols_version != op->cols->version ||
      op->pairs->rows_version != op->rows->version)
    ABX_TRY(pair_layout_build(op));
  PairLayout &L = *op->pairs;
  const int64_t nr = L.rows->n, nc = L.cols.n;
  if (nr == 0) return ABX_OK;
  if (!(L.split == matvec_split(op))) ABX_TRY(relist_units(ctx, L, matvec_split(op)));
  const bool mixed = op->precision == ABX_PREC_MIXED && op->k.kind != ABX_K_SCALAR_SUM;
  if (nc > 0)
    k_gather_b<<<ceil_div(nc, TPB), TPB, 0, ctx->stream>>>(
        b, L.cols.perm.ptr, nc, mixed ? L.bk32.ptr : nullptr, mixed ? nullptr : L.bk64.ptr,
        L.counts.ptr + 4);
  ABX_CHECK_CUDA(cudaGetLastError());
  KParams P = base_params(L);
  P.kind = op->k.kind;
  P.p0 = op->k.p[0];
  P.p0f = (float)op->k.p[0];
  P.c_exp2 = (float)(-op->k.p[0] * 1.4426950408889634);
  P.fixc = fx::consts(L.unit, 1.0 / P.p0);
  P.b32 = L.bk32.ptr;
  P.b64 = L.bk64.ptr;
  P.s_col = L.sk.ptr;
  P.s_row = L.sq.ptr;
  P.c = c;
  if (nc == 0) {
    ABX_CHECK_CUDA(cudaMemsetAsync(c, 0, nr * sizeof(double), ctx->stream));
    return ABX_OK;
  }
  return launch_matvec_kind(ctx, P, mixed, L.unit.ok);
}

namespace {
__global__ void k_aos_to_soa_q(const double *__restrict__ aos, int64_t n, int dim,
                               double *__restrict__ soa) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int d = 0; d < dim; ++d) soa[(int64_t)d * n + i] = aos[i * dim + d];
}

// Exclusive prefix sum of n counts as 64-bit row pointers (n + 1 entries):
// sums of tiles, one CTA's scan of the sums, then the tiles.  (The counts were
// summed on the host before: 8 B a row out and back.)
constexpr int RP_TPB = 256, RP_ITEMS = 8, RP_TILE = RP_TPB * RP_ITEMS;
__device__ __forceinline__ int64_t block_exclusive(int64_t v, int64_t *warp_sums, int64_t &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int64_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) warp_sums[w] = incl;
  __syncthreads();
  int64_t before = 0;
  total = 0;
  for (int i = 0; i < RP_TPB / 32; ++i) {
    if (i < w) before += warp_sums[i];
    total += warp_sums[i];
  }
  __syncthreads();
  return before + incl - v;
}
__global__ void __launch_bounds__(RP_TPB) k_rp_sums(const int32_t *__restrict__ counts, int64_t n,
                                                    int64_t *__restrict__ sums) {
  __shared__ int64_t ws[RP_TPB / 32];
  int64_t s = 0;
  for (int i = 0; i < RP_ITEMS; ++i) {
    const int64_t g = (int64_t)blockIdx.x * RP_TILE + i * RP_TPB + threadIdx.x;
    if (g < n) s += counts[g];
  }
  int64_t total;
  block_exclusive(s, ws, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(RP_TPB) k_rp_scan(int64_t *__restrict__ sums, int64_t nb,
                                                    int64_t *__restrict__ last) {
  __shared__ int64_t ws[RP_TPB / 32];
  int64_t run = 0;
  for (int64_t i0 = 0; i0 < nb; i0 += RP_TPB) {
    const int64_t i = i0 + threadIdx.x;
    int64_t total;
    const int64_t ex = block_exclusive(i < nb ? sums[i] : 0, ws, total);
    if (i < nb) sums[i] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) *last = run;
}
__global__ void __launch_bounds__(RP_TPB) k_rp_write(const int32_t *__restrict__ counts, int64_t n,
                                                     const int64_t *__restrict__ sums,
                                                     int64_t *__restrict__ rowptr) {
  __shared__ int64_t ws[RP_TPB / 32];
  const int64_t base = (int64_t)blockIdx.x * RP_TILE + (int64_t)threadIdx.x * RP_ITEMS;
  int32_t c[RP_ITEMS];
  int64_t s = 0;
  for (int i = 0; i < RP_ITEMS; ++i) {
    c[i] = base + i < n ? counts[base + i] : 0;
    s += c[i];
  }
  int64_t total;
  int64_t run = sums[blockIdx.x] + block_exclusive(s, ws, total);
  for (int i = 0; i < RP_ITEMS; ++i) {
    if (base + i < n) rowptr[base + i] = run;
    run += c[i];
  }
}

__global__ void k_rowptr_to_kernel(const int64_t *__restrict__ rowptr,
                                   const uint32_t *__restrict__ perm, int64_t n,
                                   int64_t *__restrict__ rowptr_k) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  rowptr_k[k] = rowptr[perm[k]];
}

// Row pointers (W.rowptr, n + 1 entries) from the counts W.cnt, and their total
// on the host.
int rowptr_device(abx_context *ctx, SearchSpace &W, int64_t n, int64_t &nnz) {
  cudaStream_t s = ctx->stream;
  const unsigned nb = ceil_div(n, RP_TILE);
  ABX_TRY(W.rowptr.reserve(n + 1));
  ABX_TRY(W.sums.reserve(nb + 1));
  k_rp_sums<<<nb, RP_TPB, 0, s>>>(W.cnt.ptr, n, W.sums.ptr);
  k_rp_scan<<<1, RP_TPB, 0, s>>>(W.sums.ptr, nb, W.rowptr.ptr + n);
  k_rp_write<<<nb, RP_TPB, 0, s>>>(W.cnt.ptr, n, W.sums.ptr, W.rowptr.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  ABX_CHECK_CUDA(cudaMemcpyAsync(&nnz, W.rowptr.ptr + n, 8, cudaMemcpyDeviceToHost, s));
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  return ABX_OK;
}
}  // namespace

// Host memory for lists whose length is known once they are counted.
struct OwnedLists {
  bool want_dx = false;
  int64_t nnz = 0;
  void *cols = nullptr, *dx = nullptr;
  ~OwnedLists() {
    std::free(cols);
    std::free(dx);
  }
  int allocate(int64_t n, int dim) {
    nnz = n;
    cols = std::malloc((size_t)std::max<int64_t>(n, 1) * sizeof(int32_t));
    if (want_dx) dx = std::malloc((size_t)std::max<int64_t>(n, 1) * dim * sizeof(double));
    ABX_REQUIRE(cols && (dx || !want_dx), ABX_ERR_ALLOC, "no host memory for %lld neighbours", (long long)n);
    return ABX_OK;
  }
};

// Radius queries for arbitrary points (C ABI helpers).
int radius_query(abx_particles *p, int64_t nq, const double *q_host_or_dev, double r,
                 int32_t *counts_user, int64_t *rowptr_user, int32_t *cols_user, int64_t cap,
                 int lnorm, double *dx_user = nullptr, OwnedLists *own = nullptr) {
  abx_context *ctx = p->ctx;
  cudaStream_t s = ctx->stream;
  ABX_REQUIRE(p->searchable, ABX_ERR_STATE, "init_neighbour_search not called on this particle set");
  ABX_REQUIRE(r >= 0 && std::isfinite(r), ABX_ERR_INVALID, "invalid radius");
  ABX_REQUIRE(lnorm == 2 || lnorm == 1 || lnorm == -1, ABX_ERR_INVALID,
              "norm %d not supported (2 euclidean, 1 manhattan, -1 chebyshev)", lnorm);
  const int D = p->dim;
  std::lock_guard<std::mutex> hold(p->search->m);
  SearchSpace &W = *p->search;
  const void *qd;
  ABX_TRY(W.queries.in(ctx, q_host_or_dev, (size_t)nq * D * sizeof(double), &qd));
  PairLayout &L = W.L;
  ABX_TRY(W.qsoa.reserve((size_t)D * (nq ? nq : 1)));
  if (nq)
    k_aos_to_soa_q<<<ceil_div(nq, TPB), TPB, 0, s>>>((const double *)qd, nq, D, W.qsoa.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  ABX_TRY(layout_build(ctx, p, r, W.qsoa.ptr, nq, nq, L, SPLIT_COUNT, lnorm));
  if (nq == 0) {
    if (rowptr_user) {
      int64_t z = 0;
      ABX_CHECK_CUDA(cudaMemcpy(rowptr_user, &z, sizeof(int64_t), cudaMemcpyDefault));
    }
    if (own) ABX_TRY(own->allocate(0, D));
    return ABX_OK;
  }
  // counts go by row, straight to the caller's device memory where it is that
  const bool direct = counts_user && !rowptr_user && device_ptr_usable(counts_user, ctx->device) == 1;
  int32_t *cnt = counts_user;
  if (!direct) {
    ABX_TRY(W.cnt.reserve(nq + 1));
    cnt = W.cnt.ptr;
  }
  KParams P = base_params(L);
  P.kind = ABX_K_CONST;
  P.lnorm = lnorm;
  P.thr = lnorm == 2 ? r * r : std::fabs(r);
  P.counts_out = cnt;
  if (p->n > 0)
    ABX_TRY(launch_search<POL_COUNT>(ctx, P));
  else
    ABX_CHECK_CUDA(cudaMemsetAsync(cnt, 0, nq * 4, s));
  if (counts_user && !direct)
    ABX_CHECK_CUDA(cudaMemcpyAsync(counts_user, cnt, nq * 4, cudaMemcpyDefault, s));
  if (rowptr_user) {
    int64_t nnz = 0;
    ABX_TRY(rowptr_device(ctx, W, nq, nnz));
    ABX_CHECK_CUDA(cudaMemcpyAsync(rowptr_user, W.rowptr.ptr, (nq + 1) * 8, cudaMemcpyDefault, s));
    if (own) {
      ABX_TRY(own->allocate(nnz, D));
      cols_user = static_cast<int32_t *>(own->cols);
      dx_user = static_cast<double *>(own->dx);
      cap = nnz;
    }
    if (cols_user) {
      ABX_REQUIRE(cap >= nnz, ABX_ERR_CAPACITY, "cols capacity %lld < nnz %lld", (long long)cap,
                  (long long)nnz);
      ABX_TRY(W.rpk.reserve(nq));
      ABX_TRY(W.cols.reserve(nnz ? nnz : 1));
      if (dx_user) {
        ABX_TRY(W.dxd.reserve((size_t)(nnz ? nnz : 1) * D));
        P.dx_out = W.dxd.ptr;
      }
      k_rowptr_to_kernel<<<ceil_div(nq, TPB), TPB, 0, s>>>(W.rowptr.ptr, L.rows->perm.ptr, nq,
                                                           W.rpk.ptr);
      ABX_CHECK_CUDA(cudaGetLastError());
      P.rowptr = W.rpk.ptr;
      P.cols_out = W.cols.ptr;
      if (p->n > 0 && nnz > 0) ABX_TRY(launch_search<POL_LIST>(ctx, P));
      ABX_CHECK_CUDA(cudaMemcpyAsync(cols_user, W.cols.ptr, nnz * 4, cudaMemcpyDefault, s));
      if (dx_user && nnz)
        ABX_CHECK_CUDA(cudaMemcpyAsync(dx_user, W.dxd.ptr, (size_t)nnz * D * 8, cudaMemcpyDefault, s));
    }
  }
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  W.trim(nq, p->n);
  return ABX_OK;
}

// Storage-order CSR of the neighbour lists of a particle set with itself at
// radius r (device arrays; used by the exact least-squares SPAI rows).
int self_csr_device(abx_particles *p, double r, DevBuf<int64_t> &rowptr, DevBuf<int32_t> &cols,
                    int64_t &nnz) {
  abx_context *ctx = p->ctx;
  cudaStream_t s = ctx->stream;
  const int64_t n = p->n;
  std::lock_guard<std::mutex> hold(p->search->m);
  SearchSpace &W = *p->search;
  PairLayout &L = W.L;
  ABX_TRY(layout_build(ctx, p, r, nullptr, n, n, L, SPLIT_COUNT));
  ABX_TRY(rowptr.reserve(n + 1));
  nnz = 0;
  if (n == 0) {
    ABX_CHECK_CUDA(cudaMemsetAsync(rowptr.ptr, 0, 8, s));
    return cols.reserve(1);
  }
  ABX_TRY(W.cnt.reserve(n + 1));
  KParams P = base_params(L);
  P.kind = ABX_K_CONST;
  P.counts_out = W.cnt.ptr;
  ABX_TRY(launch_search<POL_COUNT>(ctx, P));
  ABX_TRY(rowptr_device(ctx, W, n, nnz));
  ABX_CHECK_CUDA(cudaMemcpyAsync(rowptr.ptr, W.rowptr.ptr, (n + 1) * 8, cudaMemcpyDeviceToDevice, s));
  ABX_TRY(cols.reserve(nnz + 1));
  if (nnz > 0) {
    ABX_TRY(W.rpk.reserve(n));
    k_rowptr_to_kernel<<<ceil_div(n, TPB), TPB, 0, s>>>(W.rowptr.ptr, L.rows->perm.ptr, n, W.rpk.ptr);
    P.rowptr = W.rpk.ptr;
    P.cols_out = cols.ptr;
    ABX_TRY(launch_search<POL_LIST>(ctx, P));
    ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  }
  return ABX_OK;
}

namespace {
constexpr int KNN_MAX = 64;

// k nearest neighbours (FP64 distance with periodic images, ties broken by
// storage index) of every particle of the layout's column set, by rings of
// fine cells around the particle's anchor cell.  One thread per particle.
__global__ void k_knn(KParams P, int k, int64_t n, int32_t *__restrict__ idx_out,
                      double *__restrict__ d2_out) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const FineGrid &fg = P.fg;
  double bd[KNN_MAX];
  int bi[KNN_MAX];
  int cnt = 0;
  const int4 qc = P.qcell[q];
  const D4 xq = P.qpos[q];
  const int c[3] = {qc.x, qc.y, qc.z};
  const double qx[3] = {xq.x, xq.y, xq.z};
  double hmin = 1e300;
  int Rmax = 0;
  for (int e = 0; e < 3; ++e) {
    if (e < fg.eoff) continue;
    hmin = fmin(hmin, fg.h[e]);
    Rmax = max(Rmax, fg.m[e]);
  }
  for (int R = 0; R <= Rmax; ++R) {
    for (int o0 = -R; o0 <= R; ++o0) {
      if (fg.m[0] == 1 && o0 != 0) continue;
      for (int o1 = -R; o1 <= R; ++o1) {
        if (fg.m[1] == 1 && o1 != 0) continue;
        const bool edge01 = (abs(o0) == R) || (abs(o1) == R);
        for (int o2 = -R; o2 <= R; o2 += (edge01 ? 1 : max(2 * R, 1))) {
          int u[3] = {c[0] + o0, c[1] + o1, c[2] + o2}, img[3] = {0, 0, 0};
          bool ok = true;
          for (int e = 0; e < 3; ++e) {
            if (u[e] >= 0 && u[e] < fg.m[e]) continue;
            if (!fg.periodic[e] || u[e] < -fg.m[e] || u[e] >= 2 * fg.m[e]) { ok = false; break; }
            if (u[e] < 0) { u[e] += fg.m[e]; img[e] = 1; } else { u[e] -= fg.m[e]; img[e] = -1; }
          }
          if (!ok) continue;
          const uint32_t cell = ((uint32_t)u[0] * fg.m[1] + u[1]) * fg.m[2] + u[2];
          const uint32_t b = P.cell_start[cell], e = P.cell_start[cell + 1];
          for (uint32_t j = b; j < e; ++j) {
            const double d2 = exact_d2(xq, P.cpos[j], img, fg);
            const int sj = (int)P.cperm[j];
            if (cnt == k && (d2 > bd[k - 1] || (d2 == bd[k - 1] && sj > bi[k - 1]))) continue;
            int pos = cnt < k ? cnt++ : k - 1;
            while (pos > 0 && (bd[pos - 1] > d2 || (bd[pos - 1] == d2 && bi[pos - 1] > sj))) {
              bd[pos] = bd[pos - 1];
              bi[pos] = bi[pos - 1];
              --pos;
            }
            bd[pos] = d2;
            bi[pos] = sj;
          }
        }
      }
    }
    // every point of ring R+1 or beyond is at least R*h away
    const double reach = fmax(R * hmin * (1.0 - 1e-9), 0.0);
    if (cnt == k && bd[k - 1] <= reach * reach) break;
  }
  const int64_t row = P.cperm[q];
  for (int j = 0; j < k; ++j) {
    idx_out[row * k + j] = j < cnt ? bi[j] : -1;
    if (d2_out) d2_out[row * k + j] = j < cnt ? bd[j] : -1.0;
  }
  (void)qx;
}
}  // namespace

int knn_device(abx_particles *p, int k, int32_t *idx, double *d2) {
  abx_context *ctx = p->ctx;
  ABX_REQUIRE(k >= 1 && k <= KNN_MAX, ABX_ERR_INVALID, "k must be in 1..%d", KNN_MAX);
  GridDesc g;
  ABX_TRY(particles_grid_desc(p, &g));
  const int64_t n = p->n;
  if (n == 0) return ABX_OK;
  double vol = 1.0;
  for (int d = 0; d < p->dim; ++d) vol *= g.hi[d] - g.lo[d];
  const double h = std::pow(std::max(1.0, k / 4.0) * vol / (double)n, 1.0 / p->dim);
  std::lock_guard<std::mutex> hold(p->search->m);
  PairLayout &L = p->search->L;
  ABX_TRY(layout_build(ctx, p, 3.0 * h, nullptr, n, n, L, SPLIT_NONE, 2, false));
  KParams P = base_params(L);
  k_knn<<<ceil_div(n, 128), 128, 0, ctx->stream>>>(P, k, n, idx, d2);
  ABX_CHECK_CUDA(cudaGetLastError());
  ABX_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
  return ABX_OK;
}

}  // namespace abx

using namespace abx;

extern "C" {

int abx_radius_count(abx_particles *p, int64_t nq, const double *q, double r, int32_t *counts) {
  return abx_radius_count_lnorm(p, nq, q, r, 2, counts);
}

int abx_radius_query_csr(abx_particles *p, int64_t nq, const double *q, double r, int64_t *rowptr,
                         int32_t *cols, int64_t cap) {
  return abx_radius_query_csr_lnorm(p, nq, q, r, 2, rowptr, cols, cap);
}

int abx_radius_query_csr_dx(abx_particles *p, int64_t nq, const double *q, double r,
                            int64_t *rowptr, int32_t *cols, double *dx, int64_t cap) {
  ABX_REQUIRE(p && (q || nq == 0) && rowptr, ABX_ERR_INVALID, "null argument");
  ABX_TRY(ctx_activate(p->ctx));
  return radius_query(p, nq, q, r, nullptr, rowptr, cols, cap, 2, cols ? dx : nullptr);
}

int abx_radius_count_lnorm(abx_particles *p, int64_t nq, const double *q, double r, int lnorm,
                           int32_t *counts) {
  ABX_REQUIRE(p && (q || nq == 0) && (counts || nq == 0), ABX_ERR_INVALID, "null argument");
  ABX_TRY(ctx_activate(p->ctx));
  return radius_query(p, nq, q, r, counts, nullptr, nullptr, 0, lnorm);
}

int abx_radius_query_csr_new(abx_particles *p, int64_t nq, const double *q, double r, int lnorm,
                             int64_t *rowptr, int64_t *nnz, void **cols, void **dx) {
  ABX_REQUIRE(p && (q || nq == 0) && rowptr && nnz && cols, ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(!dx || lnorm == 2, ABX_ERR_INVALID, "dx is returned by the euclidean search only");
  ABX_TRY(ctx_activate(p->ctx));
  OwnedLists own;
  own.want_dx = dx != nullptr;
  ABX_TRY(radius_query(p, nq, q, r, nullptr, rowptr, nullptr, 0, lnorm, nullptr, &own));
  *nnz = own.nnz;
  *cols = std::exchange(own.cols, nullptr);
  if (dx) *dx = std::exchange(own.dx, nullptr);
  return ABX_OK;
}

void abx_host_free(void *ptr) { std::free(ptr); }

int abx_radius_query_csr_lnorm(abx_particles *p, int64_t nq, const double *q, double r, int lnorm,
                               int64_t *rowptr, int32_t *cols, int64_t cap) {
  ABX_REQUIRE(p && (q || nq == 0) && rowptr, ABX_ERR_INVALID, "null argument");
  ABX_TRY(ctx_activate(p->ctx));
  return radius_query(p, nq, q, r, nullptr, rowptr, cols, cap, lnorm);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Searches in a linearly transformed coordinate system (euclidean_search with
// a LinearTransform / ScaleTransform, src/Transform.h, src/Search.h:438-445):
// a particle is a neighbour iff !(|T dx|^2 > r^2), dx = x_j - (x + image*L).
// The candidates come from the ordinary search at radius r / sigma_min(T)
// (every point with |T dx| <= r has |dx| <= r / sigma_min), widened by 1e-9
// relative; the transformed test then runs on the device per candidate.
namespace abx {
namespace {
struct TMat {
  double m[9];  // row-major D x D
};

// (T dx)_i = ((T_i0 dx_0 + T_i1 dx_1) + T_i2 dx_2); accum = ((0 + y_0^2) + y_1^2) + y_2^2
__device__ __forceinline__ bool tf_inside(const double *dx, int D, const TMat &T, double r2,
                                          double *y) {
  double acc = 0.0;
  for (int i = 0; i < D; ++i) {
    double v = 0.0;
    for (int k = 0; k < D; ++k) v = __dadd_rn(v, __dmul_rn(T.m[i * D + k], dx[k]));
    y[i] = v;
    acc = __dadd_rn(acc, __dmul_rn(v, v));
  }
  return !(acc > r2);
}

__global__ void k_tf_count(const int64_t *__restrict__ rp, const double *__restrict__ dx,
                           int64_t nq, int D, TMat T, double r2, int64_t *__restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  int64_t c = 0;
  double y[3];
  for (int64_t e = rp[i]; e < rp[i + 1]; ++e) c += tf_inside(dx + e * D, D, T, r2, y) ? 1 : 0;
  cnt[i] = c;
}

__global__ void k_tf_fill(const int64_t *__restrict__ rp, const int32_t *__restrict__ cols,
                          const double *__restrict__ dx, int64_t nq, int D, TMat T, double r2,
                          const int64_t *__restrict__ orp, int32_t *__restrict__ ocols,
                          double *__restrict__ odx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  int64_t o = orp[i];
  double y[3];
  for (int64_t e = rp[i]; e < rp[i + 1]; ++e) {
    if (!tf_inside(dx + e * D, D, T, r2, y)) continue;
    ocols[o] = cols[e];
    if (odx)
      for (int d = 0; d < D; ++d) odx[o * D + d] = y[d];
    ++o;
  }
}

// smallest singular value of the D x D matrix T: the square root of the
// smallest eigenvalue of T^T T, by cyclic Jacobi rotations
double sigma_min(const double *T, int D) {
  double A[3][3] = {};
  for (int i = 0; i < D; ++i)
    for (int j = 0; j < D; ++j)
      for (int k = 0; k < D; ++k) A[i][j] += T[k * D + i] * T[k * D + j];
  for (int sweep = 0; sweep < 64; ++sweep) {
    double off = 0.0;
    for (int i = 0; i < D; ++i)
      for (int j = i + 1; j < D; ++j) off += A[i][j] * A[i][j];
    if (off <= 1e-300) break;
    for (int p = 0; p < D; ++p)
      for (int q = p + 1; q < D; ++q) {
        if (A[p][q] == 0.0) continue;
        const double th = 0.5 * (A[q][q] - A[p][p]) / A[p][q];
        const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < D; ++k) {  // A <- A J
          const double akp = A[k][p], akq = A[k][q];
          A[k][p] = c * akp - s * akq;
          A[k][q] = s * akp + c * akq;
        }
        for (int k = 0; k < D; ++k) {  // A <- J^T A
          const double apk = A[p][k], aqk = A[q][k];
          A[p][k] = c * apk - s * aqk;
          A[q][k] = s * apk + c * aqk;
        }
      }
  }
  double lmin = A[0][0];
  for (int i = 1; i < D; ++i) lmin = std::min(lmin, A[i][i]);
  return lmin > 0 ? std::sqrt(lmin) : 0.0;
}
}  // namespace
}  // namespace abx

// Unique pairs within r of one particle set: the pairs a sweep over
// neighbouring buckets visits (bucket_pair_iterator, src/Search.h:498-764,
// together with the pairs inside each bucket), each once -- (i, j) with i < j
// in storage order, dx = x_j - (x_i + image*L) of the accepted image and
// !(|dx|^2 > r^2) -- from the self search's CSR, filtered on the device.
namespace abx {
namespace {
__global__ void k_soa_to_aos(const double *__restrict__ soa, int64_t n, int dim,
                             double *__restrict__ aos) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int d = 0; d < dim; ++d) aos[i * dim + d] = soa[(int64_t)d * n + i];
}

__global__ void k_upper_count(const int64_t *__restrict__ rp, const int32_t *__restrict__ cols,
                              int64_t n, int64_t *__restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t c = 0;
  for (int64_t e = rp[i]; e < rp[i + 1]; ++e) c += cols[e] > i ? 1 : 0;
  cnt[i] = c;
}

__global__ void k_upper_fill(const int64_t *__restrict__ rp, const int32_t *__restrict__ cols,
                             const double *__restrict__ dx, int64_t n, int D,
                             const int64_t *__restrict__ orp, int32_t *__restrict__ oi,
                             int32_t *__restrict__ oj, double *__restrict__ odx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t o = orp[i];
  for (int64_t e = rp[i]; e < rp[i + 1]; ++e) {
    if (cols[e] <= i) continue;
    oi[o] = (int32_t)i;
    oj[o] = cols[e];
    if (odx)
      for (int d = 0; d < D; ++d) odx[o * D + d] = dx[e * D + d];
    ++o;
  }
}
}  // namespace
}  // namespace abx

extern "C" int abx_radius_pairs(abx_particles *p, double r, int64_t *npairs, int32_t *pi,
                                int32_t *pj, double *dx, int64_t cap) {
  ABX_REQUIRE(p && npairs, ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(r >= 0 && std::isfinite(r), ABX_ERR_INVALID, "invalid radius");
  ABX_REQUIRE(p->searchable, ABX_ERR_STATE, "init_neighbour_search not called on this particle set");
  ABX_TRY(ctx_activate(p->ctx));
  abx_context *ctx = p->ctx;
  cudaStream_t s = ctx->stream;
  const int64_t n = p->n;
  const int D = p->dim;
  *npairs = 0;
  if (n == 0) return ABX_OK;
  DevBuf<double> aos;
  ABX_TRY(aos.reserve((size_t)n * D));
  k_soa_to_aos<<<ceil_div(n, TPB), TPB, 0, s>>>(p->pos.ptr, n, D, aos.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  std::vector<int64_t> hc(n + 1);
  ABX_TRY(radius_query(p, n, aos.ptr, r, nullptr, hc.data(), nullptr, 0, 2));
  const int64_t nc = hc[n];
  DevBuf<int64_t> crp, cnt, orp;
  DevBuf<int32_t> ccols;
  DevBuf<double> cdx;
  ABX_TRY(crp.reserve(n + 1));
  ABX_TRY(cnt.reserve(n + 1));
  ABX_TRY(ccols.reserve(nc + 1));
  if (dx) ABX_TRY(cdx.reserve((size_t)(nc + 1) * D));
  ABX_TRY(radius_query(p, n, aos.ptr, r, nullptr, crp.ptr, ccols.ptr, nc, 2,
                       dx ? cdx.ptr : nullptr));
  k_upper_count<<<ceil_div(n, TPB), TPB, 0, s>>>(crp.ptr, ccols.ptr, n, cnt.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  std::vector<int64_t> h(n + 1);
  ABX_CHECK_CUDA(cudaMemcpyAsync(h.data(), cnt.ptr, n * 8, cudaMemcpyDeviceToHost, s));
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  int64_t run = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int64_t c = h[i];
    h[i] = run;
    run += c;
  }
  h[n] = run;
  *npairs = run;
  if (!pi) return ABX_OK;
  ABX_REQUIRE(pj, ABX_ERR_INVALID, "pi and pj are both given or both NULL");
  ABX_REQUIRE(cap >= run, ABX_ERR_CAPACITY, "pair capacity %lld < %lld pairs", (long long)cap,
              (long long)run);
  DevBuf<int32_t> oi, oj;
  DevBuf<double> odx;
  ABX_TRY(oi.reserve(run + 1));
  ABX_TRY(oj.reserve(run + 1));
  if (dx) ABX_TRY(odx.reserve((size_t)(run + 1) * D));
  ABX_TRY(orp.reserve(n + 1));
  ABX_CHECK_CUDA(cudaMemcpyAsync(orp.ptr, h.data(), (n + 1) * 8, cudaMemcpyHostToDevice, s));
  k_upper_fill<<<ceil_div(n, TPB), TPB, 0, s>>>(crp.ptr, ccols.ptr, dx ? cdx.ptr : nullptr, n, D,
                                                orp.ptr, oi.ptr, oj.ptr, dx ? odx.ptr : nullptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  if (run) {
    ABX_CHECK_CUDA(cudaMemcpyAsync(pi, oi.ptr, run * 4, cudaMemcpyDefault, s));
    ABX_CHECK_CUDA(cudaMemcpyAsync(pj, oj.ptr, run * 4, cudaMemcpyDefault, s));
    if (dx) ABX_CHECK_CUDA(cudaMemcpyAsync(dx, odx.ptr, (size_t)run * D * 8, cudaMemcpyDefault, s));
  }
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  return ABX_OK;
}

extern "C" int abx_radius_query_csr_transform(abx_particles *p, int64_t nq, const double *q,
                                              double r, const double *T, int64_t *rowptr,
                                              int32_t *cols, double *dx, int64_t cap) {
  ABX_REQUIRE(p && (q || nq == 0) && rowptr && T, ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(r >= 0 && std::isfinite(r), ABX_ERR_INVALID, "invalid radius");
  ABX_TRY(ctx_activate(p->ctx));
  const int D = p->dim;
  TMat tm{};
  for (int k = 0; k < D * D; ++k) {
    ABX_REQUIRE(std::isfinite(T[k]), ABX_ERR_INVALID, "transform entries must be finite");
    tm.m[k] = T[k];
  }
  const double smin = sigma_min(T, D);
  ABX_REQUIRE(smin > 0 && std::isfinite(r / smin), ABX_ERR_INVALID,
              "the transform must be invertible (smallest singular value %g)", smin);
  const double R = r / smin * (1.0 + 1e-9);
  abx_context *ctx = p->ctx;
  cudaStream_t s = ctx->stream;
  // candidates: CSR with the accepted image's dx, on the device
  std::vector<int64_t> hc(nq + 1);
  ABX_TRY(radius_query(p, nq, q, R, nullptr, hc.data(), nullptr, 0, 2));
  const int64_t nc = hc[nq];
  DevBuf<int64_t> crp, cnt, orp;
  DevBuf<int32_t> ccols;
  DevBuf<double> cdx;
  ABX_TRY(crp.reserve(nq + 1));
  ABX_TRY(cnt.reserve(nq + 1));
  ABX_TRY(ccols.reserve(nc + 1));
  ABX_TRY(cdx.reserve((size_t)(nc + 1) * D));
  ABX_TRY(radius_query(p, nq, q, R, nullptr, crp.ptr, ccols.ptr, nc, 2, cdx.ptr));
  if (nq)
    k_tf_count<<<ceil_div(nq, TPB), TPB, 0, s>>>(crp.ptr, cdx.ptr, nq, D, tm, r * r, cnt.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  std::vector<int64_t> h(nq + 1);
  if (nq) ABX_CHECK_CUDA(cudaMemcpyAsync(h.data(), cnt.ptr, nq * 8, cudaMemcpyDeviceToHost, s));
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  int64_t run = 0;
  for (int64_t i = 0; i < nq; ++i) {
    const int64_t c = h[i];
    h[i] = run;
    run += c;
  }
  h[nq] = run;
  ABX_CHECK_CUDA(cudaMemcpy(rowptr, h.data(), (nq + 1) * 8, cudaMemcpyDefault));
  if (!cols) return ABX_OK;
  ABX_REQUIRE(cap >= run, ABX_ERR_CAPACITY, "cols capacity %lld < nnz %lld", (long long)cap,
              (long long)run);
  DevBuf<int32_t> ocols;
  DevBuf<double> odx;
  ABX_TRY(ocols.reserve(run + 1));
  if (dx) ABX_TRY(odx.reserve((size_t)(run + 1) * D));
  ABX_TRY(orp.reserve(nq + 1));
  ABX_CHECK_CUDA(cudaMemcpyAsync(orp.ptr, h.data(), (nq + 1) * 8, cudaMemcpyHostToDevice, s));
  if (nq)
    k_tf_fill<<<ceil_div(nq, TPB), TPB, 0, s>>>(crp.ptr, ccols.ptr, cdx.ptr, nq, D, tm, r * r,
                                                 orp.ptr, ocols.ptr, dx ? odx.ptr : nullptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  if (run) {
    ABX_CHECK_CUDA(cudaMemcpyAsync(cols, ocols.ptr, run * 4, cudaMemcpyDefault, s));
    if (dx) ABX_CHECK_CUDA(cudaMemcpyAsync(dx, odx.ptr, (size_t)run * D * 8, cudaMemcpyDefault, s));
  }
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  return ABX_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free sparse matvec (abx_operator_matvec_noalloc).
//
// Some callers cannot call cudaMalloc while they apply an operator: code that
// runs under a device-memory budget owned by another runtime (a framework
// with its own caching allocator, a solver embedded in a simulation that
// pre-sizes everything at start-up), or a time-stepping loop that must not
// pay cudaMalloc/cudaFree's implicit device-wide synchronisation.  For them
// this entry point keeps the per-call scratch of the sparse matvec -- b
// gathered into the operator's internal order and the work counters of the pair
// kernels -- in one file-scope device array of fixed size instead of in buffers
// owned by the operator.  Every GPU that loads the library holds this array
// until the process exits.
namespace abx {
namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = size_t(32) << 20;  // 32 MiB
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

std::mutex g_noalloc_mutex;
unsigned char *g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// Device address of g_noalloc_scratch on `device` (current), looked up once
// per device.  In host code the symbol itself is only a host-side stand-in,
// so kernels must be given this address, never the symbol.
int noalloc_scratch(int device, unsigned char **out) {
  ABX_REQUIRE(device >= 0 && device < NOALLOC_MAX_DEVICES, ABX_ERR_INVALID,
              "device %d beyond the allocation-free entry point's table", device);
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_addr[device]) {
    void *p = nullptr;
    ABX_CHECK_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_addr[device] = (unsigned char *)p;
  }
  *out = g_noalloc_addr[device];
  return ABX_OK;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace
}  // namespace abx

extern "C" int abx_operator_matvec_noalloc(abx_operator *op, const double *b, double *c) {
  ABX_REQUIRE(op, ABX_ERR_INVALID, "null operator");
  ABX_REQUIRE(op->kind == 0, ABX_ERR_INVALID,
              "abx_operator_matvec_noalloc: only sparse operators are supported");
  const int64_t nr = op->rows->n, nc = op->cols->n;
  ABX_REQUIRE((b || nc == 0) && (c || nr == 0), ABX_ERR_INVALID, "null vector");
  abx_context *ctx = op->rows->ctx;
  ABX_TRY(ctx_activate(ctx));
  ABX_REQUIRE(op->cols->searchable, ABX_ERR_STATE,
              "init_neighbour_search not called on the column particle set");
  // A stale layout would have to be rebuilt, which allocates: refuse.
  ABX_REQUIRE(op->pairs && op->pairs->cols_version == op->cols->version &&
                  op->pairs->rows_version == op->rows->version,
              ABX_ERR_STATE,
              "abx_operator_matvec_noalloc: the particle sets changed since the operator was "
              "built; rebuild it (or call abx_operator_matvec once) before calling this");
  ABX_REQUIRE((nc == 0 || device_ptr_usable(b, ctx->device) == 1) &&
                  (nr == 0 || device_ptr_usable(c, ctx->device) == 1),
              ABX_ERR_INVALID,
              "abx_operator_matvec_noalloc: b and c must be device memory of the context's "
              "GPU (host vectors would need staging buffers)");
  if (nr == 0) return ABX_OK;
  const bool mixed = op->precision == ABX_PREC_MIXED && op->k.kind != ABX_K_SCALAR_SUM;
  const size_t need = align256((size_t)nc * (mixed ? sizeof(float) : sizeof(double))) +
                      align256((size_t)nr * sizeof(double)) + 256;
  ABX_REQUIRE(need <= NOALLOC_SCRATCH_BYTES, ABX_ERR_CAPACITY,
              "abx_operator_matvec_noalloc: needs %zu bytes of scratch (%lld rows, %lld "
              "columns) but the fixed array holds %zu bytes",
              need, (long long)nr, (long long)nc, NOALLOC_SCRATCH_BYTES);
  unsigned char *base = nullptr;
  ABX_TRY(noalloc_scratch(ctx->device, &base));
  const size_t bbytes = align256((size_t)nc * (mixed ? sizeof(float) : sizeof(double)));
  void *bk = base;
  // (8 B a row held the result before it was written in place: the limit stays)
  int *counter = (int *)(base + bbytes + align256((size_t)nr * sizeof(double)));
  cudaStream_t s = ctx->stream;
  PairLayout &L = *op->pairs;
  // (precision changed since: the units are listed anew, in the same buffers)
  if (!(L.split == matvec_split(op))) ABX_TRY(relist_units(ctx, L, matvec_split(op)));
  if (nc == 0) {
    ABX_CHECK_CUDA(cudaMemsetAsync(c, 0, nr * sizeof(double), s));
    return ABX_OK;
  }
  k_gather_b<<<ceil_div(nc, TPB), TPB, 0, s>>>(b, L.cols.perm.ptr, nc,
                                               mixed ? (float *)bk : nullptr,
                                               mixed ? nullptr : (double *)bk, counter);
  ABX_CHECK_CUDA(cudaGetLastError());
  KParams P = base_params(L);
  P.kind = op->k.kind;
  P.p0 = op->k.p[0];
  P.p0f = (float)op->k.p[0];
  P.c_exp2 = (float)(-op->k.p[0] * 1.4426950408889634);
  P.fixc = fx::consts(L.unit, 1.0 / P.p0);
  P.b32 = mixed ? (const float *)bk : nullptr;
  P.b64 = mixed ? nullptr : (const double *)bk;
  P.s_col = L.sk.ptr;
  P.s_row = L.sq.ptr;
  P.c = c;
  P.counter = counter;  // zeroed by the gather
  return launch_matvec_kind(ctx, P, mixed, L.unit.ok);
}

extern "C" int abx_knn(abx_particles *p, int k, int32_t *idx, double *d2) {
  ABX_REQUIRE(p && (idx || p->n == 0), ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(p->searchable, ABX_ERR_STATE, "init_neighbour_search not called on this particle set");
  ABX_TRY(ctx_activate(p->ctx));
  const int64_t n = p->n;
  HostStage si, sd;
  void *di, *dd = nullptr;
  ABX_TRY(si.out(p->ctx, idx, (size_t)n * k * 4, &di));
  if (d2) ABX_TRY(sd.out(p->ctx, d2, (size_t)n * k * 8, &dd));
  ABX_TRY(knn_device(p, k, (int32_t *)di, (double *)dd));
  ABX_TRY(si.finish(p->ctx, idx, (size_t)n * k * 4));
  if (d2) ABX_TRY(sd.finish(p->ctx, d2, (size_t)n * k * 8));
  return ABX_OK;
}
