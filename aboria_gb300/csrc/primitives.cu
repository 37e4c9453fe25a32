// Device primitives for the cell-list build: exclusive scan and a stable LSD
// radix sort of (u32 key, u32 value) pairs.
//
// The reference reaches these through Thrust (detail::exclusive_scan,
// detail::sort_by_key: src/detail/Algorithms.h:173-206, :551-580).  Its Thrust
// backend sorts stably (thrust::sort_by_key, :195), which is the order this
// sort reproduces: (key, input position).
//
// Layout: tiles of 4096 items (256 threads x 16).  Within a tile each warp owns
// 512 consecutive items, lane l holding items l, l+32, ... so that walking the
// 16 slots in order visits the warp's items in input order; ranking with
// __match_any_sync then gives a stable per-warp rank without a block-wide
// local sort.
#include <algorithm>
#include <utility>

#include "common.cuh"

namespace abx {

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;  // 4096

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive scan of a 4096-item tile held in shared memory; returns the tile
// total to every thread.
__device__ uint32_t block_scan_tile(uint32_t *s, uint32_t *warp_tot) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t local[SCAN_ITEMS];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    local[i] = s[tid * SCAN_ITEMS + i];
    sum += local[i];
  }
  uint32_t incl = warp_incl_scan(sum);
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (SCAN_THREADS / 32) ? warp_tot[lane] : 0;
    uint32_t wi = warp_incl_scan(w);
    if (lane < (SCAN_THREADS / 32)) warp_tot[lane] = wi - w;
    if (lane == (SCAN_THREADS / 32) - 1) warp_tot[SCAN_THREADS / 32] = wi;
  }
  __syncthreads();
  uint32_t run = warp_tot[warp] + incl - sum;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    s[tid * SCAN_ITEMS + i] = run;
    run += local[i];
  }
  uint32_t total = warp_tot[SCAN_THREADS / 32];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t *in, size_t n,
                                                              uint32_t *block_sums) {
  __shared__ uint32_t red[SCAN_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * SCAN_TILE;
  uint32_t sum = 0;
  for (int i = threadIdx.x; i < SCAN_TILE; i += SCAN_THREADS) {
    size_t g = base + i;
    if (g < n) sum += in[g];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < SCAN_THREADS / 32; ++w) t += red[w];
    block_sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(uint32_t *data, size_t n,
                                                             const uint32_t *block_offsets) {
  __shared__ uint32_t s[SCAN_TILE];
  __shared__ uint32_t warp_tot[SCAN_THREADS / 32 + 1];
  const size_t base = (size_t)blockIdx.x * SCAN_TILE;
  for (int i = threadIdx.x; i < SCAN_TILE; i += SCAN_THREADS) {
    size_t g = base + i;
    s[i] = g < n ? data[g] : 0u;
  }
  __syncthreads();
  block_scan_tile(s, warp_tot);
  const uint32_t off = block_offsets ? block_offsets[blockIdx.x] : 0u;
  for (int i = threadIdx.x; i < SCAN_TILE; i += SCAN_THREADS) {
    size_t g = base + i;
    if (g < n) data[g] = s[i] + off;
  }
}

// ---------------------------------------------------------------- radix ---
// LSD radix sort of (key, value) pairs, stable; RB-bit digits (8, or 10 when
// two 10-bit passes cover the key where 8-bit digits would need three).
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 4096
constexpr int RADIX_MAX = 1 << 10;

template <int RB>
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const uint32_t *keys, size_t n,
                                                           int shift, uint32_t mask,
                                                           uint32_t *hist, int ntiles) {
  constexpr int RADIX = 1 << RB;
  __shared__ uint32_t h[RADIX];
  for (int i = threadIdx.x; i < RADIX; i += RS_THREADS) h[i] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * RS_TILE;
  for (int i = threadIdx.x; i < RS_TILE; i += RS_THREADS) {
    size_t g = base + i;
    if (g < n) atomicAdd(&h[(keys[g] >> shift) & mask], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RADIX; d += RS_THREADS)
    hist[(size_t)d * ntiles + blockIdx.x] = h[d];
}

template <int RB>
__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(
    const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in,
    uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, size_t n, int shift,
    uint32_t mask, const uint32_t *__restrict__ offsets, int ntiles) {
  constexpr int RADIX = 1 << RB;
  __shared__ uint32_t wcount[RS_WARPS][RADIX + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < RS_WARPS * (RADIX + 1); i += RS_THREADS) (&wcount[0][0])[i] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * RS_TILE + (size_t)warp * (32 * RS_ITEMS);
  uint32_t key[RS_ITEMS], val[RS_ITEMS], rank[RS_ITEMS];
  int dig[RS_ITEMS];
  const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    size_t g = base + (size_t)i * 32 + lane;
    if (g < n) {
      key[i] = keys_in[g];
      val[i] = vals_in[g];
      dig[i] = (key[i] >> shift) & mask;
    } else {
      key[i] = 0;
      val[i] = 0;
      dig[i] = RADIX;  // sentinel bucket, never written out
    }
  }
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    const uint32_t peers = __match_any_sync(0xffffffffu, dig[i]);
    const int leader = 31 - __clz(peers);
    const uint32_t before = __popc(peers & lt_mask);
    const uint32_t cnt = wcount[warp][dig[i]];
    rank[i] = cnt + before;
    __syncwarp();
    if (lane == leader) wcount[warp][dig[i]] = cnt + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // exclusive prefix over warps, per digit
  for (int d = tid; d < RADIX; d += RS_THREADS) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      uint32_t c = wcount[w][d];
      wcount[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    if (dig[i] < RADIX) {
      const size_t dst = (size_t)offsets[(size_t)dig[i] * ntiles + blockIdx.x] +
                         wcount[warp][dig[i]] + rank[i];
      keys_out[dst] = key[i];
      vals_out[dst] = val[i];
    }
  }
}

// ---- few tiles: the digit offsets without scan launches
//
// Up to RF_MAX items a pass is two launches: counts per tile, and the scatter,
// whose CTAs each add up the whole (tile, digit) table from L2 (16-bit counts,
// 512 KB at most: 2,048 items a tile, 4,096 above 128 tiles; 16 bytes a load:
// loads of one count each, 49 tiles in a row, were two thirds of the scatter's
// time).  With so few tiles an 11-bit digit costs little, so that 22-bit keys take
// two passes.  Two independent sets (a search's queries and its particles) go
// through every launch together, blockIdx.y choosing the set: a pass over 100,000
// items occupies a third of the SMs.  N = 100,000, 21-bit keys: 3 x (hist, 3 scan
// kernels, scatter) + 2 copies -> 2 x 2 launches, 29 us a pass for two such sets
// (77 one after the other with single counts).
constexpr int RF_TILES = 128;
constexpr size_t RF_MAX = (size_t)RF_TILES * RS_TILE;
static_assert(RS_TILE < 65536, "16-bit counts per tile");
template <int RB, int ITEMS>
__global__ void __launch_bounds__(RS_THREADS) k_rf_hist(SortSides S, bool alt, int shift) {
  constexpr int RADIX = 1 << RB;
  __shared__ uint32_t h[RADIX];
  const SortSide &T = S.s[blockIdx.y];
  const size_t n = T.n, base = (size_t)blockIdx.x * (RS_THREADS * ITEMS);
  if (base >= n) return;
  const uint32_t *__restrict__ keys = alt ? T.keys_alt : T.keys;
  for (int i = threadIdx.x; i < RADIX; i += RS_THREADS) h[i] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const size_t g = base + i * RS_THREADS + threadIdx.x;
    if (g < n) atomicAdd(&h[(keys[g] >> shift) & (RADIX - 1)], 1u);
  }
  __syncthreads();
  uint32_t *row = T.temp + (size_t)blockIdx.x * (RADIX / 2);
  for (int d = threadIdx.x; d < RADIX / 2; d += RS_THREADS) row[d] = h[2 * d] | (h[2 * d + 1] << 16);
}

// Stable rank of every item of a tile among the items of its digit: warps own
// consecutive runs of 32 x ITEMS items, lane l the items l, l + 32, ... (see
// the top of this file).  wcount: [warp][RADIX + 1], zeroed.
template <int RADIX, int ITEMS, typename C>
__device__ __forceinline__ void rank_items(const int (&dig)[ITEMS], C *wc, uint32_t (&rank)[ITEMS]) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t peers = __match_any_sync(0xffffffffu, dig[i]);
    const int leader = 31 - __clz(peers);
    const uint32_t cnt = wc[dig[i]];
    rank[i] = cnt + __popc(peers & lt_mask);
    __syncwarp();
    if (lane == leader) wc[dig[i]] = (C)(cnt + __popc(peers));
    __syncwarp();
  }
}

// Zeroes the warps' digit counts.
template <int WARPS, int ROW, int THREADS>
__device__ __forceinline__ void clear_counts(uint16_t (*wc)[ROW]) {
  uint32_t *w = reinterpret_cast<uint32_t *>(&wc[0][0]);
  for (int i = threadIdx.x; i < WARPS * ROW / 2; i += THREADS) w[i] = 0;
}

// The warps' counts to the counts of the warps before, two digits a word (a
// tile's counts stay below 2^16); the totals to `total` if it is given.
template <int WARPS, int ROW, int THREADS, int RADIX>
__device__ __forceinline__ void scan_counts(uint16_t (*wc)[ROW], uint32_t *total) {
  for (int d = threadIdx.x; d < RADIX / 2; d += THREADS) {
    uint32_t run = 0;
#pragma unroll 8
    for (int w = 0; w < WARPS; ++w) {
      uint32_t *p = reinterpret_cast<uint32_t *>(&wc[w][0]) + d;
      const uint32_t c = *p;
      *p = run;
      run += c;
    }
    if (total) {
      total[2 * d] = run & 0xffffu;
      total[2 * d + 1] = run >> 16;
    }
  }
}

// Exclusive scan over the CTA of PER values a thread.
template <int PER>
__device__ __forceinline__ void scan_values(uint32_t (&v)[PER], uint32_t *warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) sum += v[k];
  const uint32_t incl = warp_incl_scan(sum);
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
  for (int w = 0; w < warp; ++w) run += warp_tot[w];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint32_t c = v[k];
    v[k] = run;
    run += c;
  }
}

template <int RB, int ITEMS>
__global__ void __launch_bounds__(RS_THREADS) k_rf_scatter(SortSides S, bool alt, int shift) {
  constexpr int RADIX = 1 << RB;
  constexpr int PER = RADIX / RS_THREADS;  // digits a thread adds up, consecutive
  constexpr int TILE = RS_THREADS * ITEMS;
  static_assert(PER == 1 || PER == 4 || PER == 8, "whole loads of 16-bit counts");
  __shared__ __align__(16) uint16_t wcount[RS_WARPS][RADIX + 2];
  __shared__ uint32_t first[RADIX];
  __shared__ uint32_t warp_tot[RS_WARPS];
  const SortSide &T = S.s[blockIdx.y];
  const size_t n = T.n;
  if ((size_t)blockIdx.x * TILE >= n) return;
  const uint32_t *__restrict__ keys_in = alt ? T.keys_alt : T.keys;
  const uint32_t *__restrict__ vals_in = alt ? T.vals_alt : T.vals;
  uint32_t *__restrict__ keys_out = alt ? T.keys : T.keys_alt;
  uint32_t *__restrict__ vals_out = alt ? T.vals : T.vals_alt;
  const bool iota = S.iota && shift == 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t base = (size_t)blockIdx.x * TILE + (size_t)warp * (32 * ITEMS);
  uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
  int dig[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const size_t g = base + (size_t)i * 32 + lane;
    key[i] = g < n ? keys_in[g] : 0u;
    val[i] = g < n ? (iota ? (uint32_t)g : vals_in[g]) : 0u;
    dig[i] = g < n ? (int)((key[i] >> shift) & (RADIX - 1)) : RADIX;  // RADIX: never written out
  }
  clear_counts<RS_WARPS, RADIX + 2, RS_THREADS>(wcount);
  // all tiles' counts of every digit, and those of the tiles before
  uint32_t tot[PER], pre[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) tot[k] = pre[k] = 0;
  const unsigned tiles = (unsigned)((n + TILE - 1) / TILE);
  const uint16_t *hist = reinterpret_cast<const uint16_t *>(T.temp) + tid * PER;
#pragma unroll 8
  for (unsigned t = 0; t < tiles; ++t) {
    const bool lower = t < blockIdx.x;
    if (PER == 1) {
      const uint32_t c = hist[(size_t)t * RADIX];
      tot[0] += c;
      pre[0] += lower ? c : 0u;
    } else {
      uint32_t w[PER / 2 ? PER / 2 : 1];
      if (PER == 8) {
        const uint4 v = *reinterpret_cast<const uint4 *>(hist + (size_t)t * RADIX);
        w[0] = v.x;
        w[1 % (PER / 2 ? PER / 2 : 1)] = v.y;
        w[2 % (PER / 2 ? PER / 2 : 1)] = v.z;
        w[3 % (PER / 2 ? PER / 2 : 1)] = v.w;
      } else {
        const uint2 v = *reinterpret_cast<const uint2 *>(hist + (size_t)t * RADIX);
        w[0] = v.x;
        w[1 % (PER / 2 ? PER / 2 : 1)] = v.y;
      }
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const uint32_t c = (k & 1) ? w[k / 2] >> 16 : w[k / 2] & 0xffffu;
        tot[k] += c;
        pre[k] += lower ? c : 0u;
      }
    }
  }
  scan_values<PER>(tot, warp_tot);
#pragma unroll
  for (int k = 0; k < PER; ++k) first[tid * PER + k] = tot[k] + pre[k];
  __syncthreads();
  rank_items<RADIX, ITEMS>(dig, wcount[warp], rank);
  __syncthreads();
  scan_counts<RS_WARPS, RADIX + 2, RS_THREADS, RADIX>(wcount, nullptr);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    if (dig[i] < RADIX) {
      const uint32_t dst = first[dig[i]] + wcount[warp][dig[i]] + rank[i];
      keys_out[dst] = key[i];
      vals_out[dst] = val[i];
    }
  }
}

// ---- one tile: all passes in one launch, a CTA a set, the items in shared
// memory between them.
constexpr int R1_THREADS = 512, R1_ITEMS = 8, R1_TILE = R1_THREADS * R1_ITEMS, R1_RB = 8;
template <int ITEMS>
__global__ void __launch_bounds__(R1_THREADS) k_r1_sort(SortSides S, int bits) {
  constexpr int RADIX = 1 << R1_RB, WARPS = R1_THREADS / 32;
  __shared__ uint32_t sk[R1_THREADS * ITEMS], sv[R1_THREADS * ITEMS];
  __shared__ __align__(16) uint16_t wcount[WARPS][RADIX + 2];
  __shared__ uint32_t first[RADIX], warp_tot[WARPS];
  const SortSide &T = S.s[blockIdx.x];
  const int n = (int)T.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
  int dig[ITEMS];
  for (int shift = 0; shift < bits; shift += R1_RB) {
    clear_counts<WARPS, RADIX + 2, R1_THREADS>(wcount);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = warp * (32 * ITEMS) + i * 32 + lane;
      const bool in = g < n;
      if (shift == 0) {
        key[i] = in ? T.keys[g] : 0u;
        val[i] = in ? (S.iota ? (uint32_t)g : T.vals[g]) : 0u;
      } else {
        key[i] = in ? sk[g] : 0u;
        val[i] = in ? sv[g] : 0u;
      }
      dig[i] = in ? (int)((key[i] >> shift) & (RADIX - 1)) : RADIX;
    }
    __syncthreads();
    rank_items<RADIX, ITEMS>(dig, wcount[warp], rank);
    __syncthreads();
    scan_counts<WARPS, RADIX + 2, R1_THREADS, RADIX>(wcount, first);
    __syncthreads();
    uint32_t c[1] = {tid < RADIX ? first[tid] : 0u};
    scan_values<1>(c, warp_tot);
    if (tid < RADIX) first[tid] = c[0];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (dig[i] < RADIX) {
        const uint32_t dst = first[dig[i]] + wcount[warp][dig[i]] + rank[i];
        sk[dst] = key[i];
        sv[dst] = val[i];
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < n; i += R1_THREADS) {
    T.keys[i] = sk[i];
    T.vals[i] = sv[i];
  }
}

template <int RB>
void rf_pass(const SortSides &S, dim3 grid, bool small, bool alt, int shift, cudaStream_t s) {
  if (small) {
    k_rf_hist<RB, RS_ITEMS / 2><<<grid, RS_THREADS, 0, s>>>(S, alt, shift);
    k_rf_scatter<RB, RS_ITEMS / 2><<<grid, RS_THREADS, 0, s>>>(S, alt, shift);
  } else {
    k_rf_hist<RB, RS_ITEMS><<<grid, RS_THREADS, 0, s>>>(S, alt, shift);
    k_rf_scatter<RB, RS_ITEMS><<<grid, RS_THREADS, 0, s>>>(S, alt, shift);
  }
}

__global__ void k_sort_iota(uint32_t *v, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = (uint32_t)i;
}

}  // namespace

size_t scan_temp_elems(size_t n) {
  size_t total = 0;
  size_t m = n;
  while (m > (size_t)SCAN_TILE) {
    m = (m + SCAN_TILE - 1) / SCAN_TILE;
    total += m + 64;  // padding keeps levels apart
  }
  return total + 64;
}

int exclusive_scan_u32(uint32_t *data, size_t n, uint32_t *temp, cudaStream_t s) {
  if (n == 0) return ABX_OK;
  if (n <= (size_t)SCAN_TILE) {
    k_scan_tiles<<<1, SCAN_THREADS, 0, s>>>(data, n, nullptr);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  const size_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  uint32_t *sums = temp;
  k_scan_reduce<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(data, n, sums);
  ABX_CHECK_CUDA(cudaGetLastError());
  ABX_TRY(exclusive_scan_u32(sums, nb, temp + nb + 64, s));
  k_scan_tiles<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(data, n, sums);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

size_t radix_temp_u32(size_t n) {
  const size_t ntiles = (n + RS_TILE - 1) / RS_TILE;
  const size_t hist = ntiles * RADIX_MAX;
  // (the passes over few tiles: 2048 digits)
  return std::max(hist + 64 + scan_temp_elems(hist), std::min<size_t>(2 * ntiles, RF_TILES) * 1024 + 4);
}

bool radix_few_tiles(size_t n) { return n <= RF_MAX; }

int radix_sort_sides(SortSides S, int bits, cudaStream_t s) {
  size_t most = 0;
  for (int i = 0; i < S.sides; ++i) most = std::max(most, S.s[i].n);
  const int passes = (bits + 10) / 11;
  if (most == 0) return ABX_OK;
  if (!radix_few_tiles(most) || bits <= 0) {
    for (int i = 0; i < S.sides; ++i) {
      const SortSide &T = S.s[i];
      if (S.iota && T.n) k_sort_iota<<<(unsigned)((T.n + 255) / 256), 256, 0, s>>>(T.vals, T.n);
      ABX_TRY(radix_sort_pairs(T.keys, T.vals, T.n, bits, T.keys_alt, T.vals_alt, T.temp, s));
    }
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  if (most <= (size_t)R1_TILE) {
    if (most <= R1_TILE / 4)
      k_r1_sort<R1_ITEMS / 4><<<S.sides, R1_THREADS, 0, s>>>(S, bits);
    else if (most <= R1_TILE / 2)
      k_r1_sort<R1_ITEMS / 2><<<S.sides, R1_THREADS, 0, s>>>(S, bits);
    else
      k_r1_sort<R1_ITEMS><<<S.sides, R1_THREADS, 0, s>>>(S, bits);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  const bool small = most <= RF_MAX / 2;
  const int tile = small ? RS_TILE / 2 : RS_TILE;
  const dim3 grid((unsigned)((most + tile - 1) / tile), S.sides);
  for (int i = 0; i < S.sides; ++i)  // whole 16-byte loads (radix_temp_u32 has the room)
    S.s[i].temp = reinterpret_cast<uint32_t *>((reinterpret_cast<uintptr_t>(S.s[i].temp) + 15) & ~(uintptr_t)15);
  const int rb = (bits + passes - 1) / passes;
  bool alt = false;
  for (int shift = 0; shift < bits; shift += rb, alt = !alt) {
    if (rb <= 8)
      rf_pass<8>(S, grid, small, alt, shift, s);
    else if (rb <= 10)
      rf_pass<10>(S, grid, small, alt, shift, s);
    else
      rf_pass<11>(S, grid, small, alt, shift, s);
  }
  ABX_CHECK_CUDA(cudaGetLastError());
  for (int i = 0; alt && i < S.sides; ++i) {
    const SortSide &T = S.s[i];
    ABX_CHECK_CUDA(cudaMemcpyAsync(T.keys, T.keys_alt, T.n * 4, cudaMemcpyDeviceToDevice, s));
    ABX_CHECK_CUDA(cudaMemcpyAsync(T.vals, T.vals_alt, T.n * 4, cudaMemcpyDeviceToDevice, s));
  }
  return ABX_OK;
}

int radix_sort_pairs(uint32_t *keys, uint32_t *vals, size_t n, int bits, uint32_t *keys_alt,
                     uint32_t *vals_alt, uint32_t *temp, cudaStream_t s) {
  if (n <= 1 || bits <= 0) return ABX_OK;
  const int ntiles = (int)((n + RS_TILE - 1) / RS_TILE);
  if (radix_few_tiles(n)) {
    SortSides S{};
    S.sides = 1;
    S.s[0] = SortSide{keys, vals, keys_alt, vals_alt, temp, n};
    return radix_sort_sides(S, bits, s);
  }
  // digit width: 9 or 10 bits where that saves a pass (17..20- and 25..27-bit keys)
  const int rb = (bits > 16 && bits <= 20) ? 10 : (bits > 24 && bits <= 27) ? 9 : 8;
  const size_t hist_n = (size_t)ntiles << rb;
  uint32_t *hist = temp;
  uint32_t *scan_tmp = temp + hist_n + 64;
  uint32_t *ki = keys, *vi = vals, *ko = keys_alt, *vo = vals_alt;
  for (int shift = 0; shift < bits; shift += rb) {
    const int nb = bits - shift < rb ? bits - shift : rb;
    const uint32_t mask = (1u << nb) - 1u;
    if (rb == 10)
      k_radix_hist<10><<<ntiles, RS_THREADS, 0, s>>>(ki, n, shift, mask, hist, ntiles);
    else if (rb == 9)
      k_radix_hist<9><<<ntiles, RS_THREADS, 0, s>>>(ki, n, shift, mask, hist, ntiles);
    else
      k_radix_hist<8><<<ntiles, RS_THREADS, 0, s>>>(ki, n, shift, mask, hist, ntiles);
    ABX_CHECK_CUDA(cudaGetLastError());
    ABX_TRY(exclusive_scan_u32(hist, hist_n, scan_tmp, s));
    if (rb == 10)
      k_radix_scatter<10><<<ntiles, RS_THREADS, 0, s>>>(ki, vi, ko, vo, n, shift, mask, hist, ntiles);
    else if (rb == 9)
      k_radix_scatter<9><<<ntiles, RS_THREADS, 0, s>>>(ki, vi, ko, vo, n, shift, mask, hist, ntiles);
    else
      k_radix_scatter<8><<<ntiles, RS_THREADS, 0, s>>>(ki, vi, ko, vo, n, shift, mask, hist, ntiles);
    ABX_CHECK_CUDA(cudaGetLastError());
    uint32_t *t;
    t = ki; ki = ko; ko = t;
    t = vi; vi = vo; vo = t;
  }
  if (ki != keys) {
    ABX_CHECK_CUDA(cudaMemcpyAsync(keys, ki, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    ABX_CHECK_CUDA(cudaMemcpyAsync(vals, vi, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  }
  return ABX_OK;
}

}  // namespace abx
