// Black-box Chebyshev FMM operator (create_fmm_operator, src/Operators.h:
// 401-407; KernelFMM src/Kernels.h:533-576).
//
// Reference algorithm (restated, not translated):
//  * expansions: BlackBoxExpansions (src/detail/FastMultipoleMethod.h:96-368)
//    with Chebyshev interpolation (src/detail/Chebyshev.h:84-153, 245-294):
//    R_j(x) = prod_d S_{m_d(j)}(x_d), nodes in lattice order (last dim fastest);
//  * traversal: FastMultipoleMethod::matrix_vector_multiply
//    (src/FastMultipoleMethod.h:111-548) with theta_condition
//    (src/detail/FastMultipoleMethod.h:1249-1279), P2P at target leaves over
//    the connected list (leaf or whole subtree).
//
// GB300 design: the traversal runs once per operator (octree.cu, on the device)
// and is flattened into per-level lists (M2L pairs, P2P leaf pairs, parent/child
// links); translation operators are precomputed instead of re-evaluating the
// kernel at node pairs on every call: one M2M/L2L matrix per child octant
// (the Chebyshev interpolation is scale invariant) and one M2L matrix per
// (level, box offset) -- M2L pairs at one level differ only by an integer box
// offset in [-3, 3]^D.  Each matvec is five passes of device kernels: P2M,
// M2M (bottom-up), M2L, L2L (top-down), then L2P+P2P per target leaf.
//
// M2L runs as a GEMM per (level, offset):
//   G[:, targets] += K_o * W[:, sources]
// in the mixed-precision mode on the tensor cores with FP32 accumulation (split
// FP16 on tcgen05 above 64 nodes, 3xTF32 on mma.sync below) and P2P in FP32; in
// the FP64 mode M2L is a product of scaled 56-bit integers, by their digits on the
// tensor cores, for matrices whose rows hold values of one size, and in FP64 for the
// others; P2P takes its kernel values from the integer units (fix64.cuh).  Both have
// errors no larger than FP64's own.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <functional>
#include <map>
#include <vector>

#include <cuda_fp16.h>

#include "common.cuh"
#include "digits.cuh"
#include "fix64.cuh"
#include "handles.cuh"

namespace abx {

constexpr int MAXN_TAB = 8;  // max Chebyshev order of the coefficient table

// Clenshaw coefficients of S_m: c[m][k] = (2/n) cos(k (2m+1) pi / (2n)).
struct ChebTab {
  double c[MAXN_TAB][MAXN_TAB];
};
struct ChebTab32 {  // the same in FP32 (mixed-precision P2M and L2P)
  float c[MAXN_TAB][MAXN_TAB];
};

struct FmmPlan {
  int D = 3, n = 3, ncheb = 27, nchild = 8;
  int nnodes = 0;
  int kind = 0;
  double p0 = 0.0;
  std::vector<int> mi;  // ncheb x D multi-indices
  // device
  DevBuf<double> W, G;            // nnodes x ncheb
  DevBuf<double> Tc;              // nchild x ncheb x ncheb (child->parent interpolation)
  DevBuf<float> Tc32;             // FP32 copy (mixed-precision L2L)
  DevBuf<double> TcT;             // transposed: TcT[o][j][i] = Tc[o][i][j] (M2M)
  DevBuf<float> Tc32T;            // FP32 copy of TcT (mixed-precision M2M)
  DevBuf<double> box;             // nnodes x 6 (lo[3], hi[3])
  DevBuf<int> leaf_ids;           // leaves (node ids)
  DevBuf<int> node_begin, node_end;
  // per level: nodes with children (M2M/L2L), (parent, child, octant) links
  std::vector<int> max_level;
  std::vector<std::vector<int>> level_links;  // host: flattened (parent, child, octant)
  DevBuf<int> links;                          // all levels, octant-major within a level
  DevBuf<int2> batches;                       // (first link, count <= NBL) of one octant
  std::vector<int> batch_off, batch_cnt;      // per level
  int n_m2l = 0;
  DevBuf<double> Km;      // nmat x ncheb x ncheb
  DevBuf<float> Kmh, Kml; // split-TF32 hi/lo parts of the FP32 copy (mma.sync M2L, ncheb <= 64)
  DevBuf<__half> Kp;      // the same packed as tcgen05 stage images (ncheb > 64, k_pack_f16)
  DevBuf<float> Kp_scale;  // power of two of each matrix' packed values
  // FP64 M2L: digits of K and W, their exponents (per row of K, per node), tiles
  DevBuf<__half> Kd, Wd;
  DevBuf<short> ke, we;
  DevBuf<int> mf_mat, mf_first;  // tiles of the matrices that are multiplied by digits
  DevBuf<int> mw_mat, mw_first;  // and of those with rows of many sizes (k_m2l64)
  int mf_tiles = 0, mw_tiles = 0;
  bool m2l64_ready = false;
  // W as scaled FP16, hi and lo, and each node's power of two (tcgen05 M2L)
  DevBuf<__half> W16h, W16l;
  DevBuf<float> W16_scale;
  int nmat = 0;
  // M2L grouped by matrix (for the tensor-core GEMM): per matrix a list of
  // (target, source)
  DevBuf<int2> m2l_by_mat;
  std::vector<int> mat_off, mat_cnt;
  DevBuf<int> mat_off_d;
  // P2P: CSR over target leaves of source leaves
  DevBuf<int> p2p_rowptr, p2p_src;
  int nleaves = 0;
  double build_s = 0.0;
  double chebsetup_s = 0.0;
  // tcgen05 M2L: limit of each mbarrier wait, and the test-only fault
  // injection that withholds one operand-ready signal
  double wait_limit_s = 1.0;
  int drop_arrive = 0;
  DevBuf<float> W32, G32;
  ChebTab tab{};        // Clenshaw coefficients of the order
  ChebTab32 tab32{};    // the same in FP32 (mixed-precision P2M / L2P)
  DevBuf<float4> posf;  // mixed near field: FP32 position relative to the leaf centre
  DevBuf<float> b32;    // mixed near field: FP32 weights of the current matvec
  // FP64 near field on the integer units (fix64.cuh), where unit.ok: the
  // positions in fixed point, written by every matvec
  fx::Unit unit{};
  DevBuf<longlong2> fxy;
  DevBuf<long long> fz;
  DevBuf<int> mi_d;                 // ncheb x 3 multi-indices
  DevBuf<int> tile_mat, tile_first; // tensor-core M2L tiles
  int ntiles = 0, tile_pairs = 0;
  int sms = 1;  // of the plan's GPU
};

void fmm_plan_free(FmmPlan *P) { delete P; }

namespace {

constexpr double PI = 3.14159265358979323846;

// S_m(x), m = 0..n-1 (chebyshev_Sn: Clenshaw, src/detail/Chebyshev.h:135-153)
__host__ __device__ inline void cheb_sn(double x, int n, double *S) {
  const double invn = 1.0 / n;
  for (int m = 0; m < n; ++m) {
    double b1 = 0.0, b2 = 0.0;
    for (int k = n - 1; k >= 1; --k) {
      const double bk = 2 * invn * cos(k * (2.0 * m + 1.0) * (PI / 2) * invn) + 2.0 * x * b1 - b2;
      b2 = b1;
      b1 = bk;
    }
    S[m] = invn + x * b1 - b2;
  }
}

__host__ __device__ inline double cheb_node(int m, int n) { return cos((2.0 * m + 1.0) * PI / (2.0 * n)); }

// The Clenshaw coefficients of S_m (ChebTab, declared with the plan),
// computed once on the host (the same std::cos values as the host-side
// recurrence above) and passed by value, so that no kernel evaluates cos.
inline ChebTab cheb_table(int n) {
  ChebTab t{};
  const double invn = 1.0 / n;
  for (int m = 0; m < n; ++m)
    for (int k = 1; k < n; ++k) t.c[m][k] = 2 * invn * cos(k * (2.0 * m + 1.0) * (PI / 2) * invn);
  return t;
}

// S_m(x), m = 0..n-1, with the tabulated coefficients: the same recurrence
// as cheb_sn.
__device__ __forceinline__ void cheb_sn_tab(double x, int n, const ChebTab &t, double *S) {
  const double invn = 1.0 / n;
  for (int m = 0; m < n; ++m) {
    double b1 = 0.0, b2 = 0.0;
    for (int k = n - 1; k >= 1; --k) {
      const double bk = t.c[m][k] + 2.0 * x * b1 - b2;
      b2 = b1;
      b1 = bk;
    }
    S[m] = invn + x * b1 - b2;
  }
}

// FP32 copy of the Clenshaw coefficients and the same recurrence in FP32
// (mixed-precision P2M and L2P).

inline ChebTab32 cheb_table32(const ChebTab &t) {
  ChebTab32 f{};
  for (int m = 0; m < MAXN_TAB; ++m)
    for (int k = 0; k < MAXN_TAB; ++k) f.c[m][k] = (float)t.c[m][k];
  return f;
}

__device__ __forceinline__ void cheb_sn_tab32(float x, int n, const ChebTab32 &t, float *S) {
  const float invn = 1.0f / (float)n;
  for (int m = 0; m < n; ++m) {
    float b1 = 0.f, b2 = 0.f;
    for (int k = n - 1; k >= 1; --k) {
      const float bk = t.c[m][k] + 2.f * x * b1 - b2;
      b2 = b1;
      b1 = bk;
    }
    S[m] = invn + x * b1 - b2;
  }
}

__host__ __device__ inline double shift_coord(double p, double lo, double hi) {
  const double span = hi - lo;
  return span > 0.0 ? (2 * p - lo - hi) / span : 0.0;
}

template <int KIND> __device__ __forceinline__ double fmm_k64(double d2, double p0) {
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return exp(-d2 * p0);
  if (KIND == ABX_K_LAPLACE) return 1.0 / (sqrt(d2) + p0);
  if (KIND == ABX_K_MULTIQUADRIC) return sqrt(d2 + p0);
  if (KIND == ABX_K_CONST) return p0;
  return 0.0;
}

template <int KIND> __device__ __forceinline__ float fmm_k32(float d2, float p0) {
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return __expf(-d2 * p0);
  if (KIND == ABX_K_LAPLACE) return __fdividef(1.0f, sqrtf(d2) + p0);
  if (KIND == ABX_K_MULTIQUADRIC) return sqrtf(d2 + p0);
  if (KIND == ABX_K_CONST) return p0;
  return 0.0f;
}

// ---------------------------------------------------------------- P2M ---
constexpr int FT = 128;
constexpr int MAXN = 8;     // max Chebyshev order
constexpr int MAXC = 512;   // max nodes (8^3)

__global__ void __launch_bounds__(FT) k_p2m(int D, int n, int ncheb, const int *__restrict__ leaves,
                                            const int *__restrict__ nb, const int *__restrict__ ne,
                                            const double *__restrict__ box,
                                            const double *__restrict__ pos, int64_t npos,
                                            const double *__restrict__ b, const int *__restrict__ mi,
                                            const ChebTab tab, double *__restrict__ W) {
  __shared__ double S[FT][MAXN * 3];
  __shared__ double sb[FT];
  const int leaf = leaves[blockIdx.x];
  const double *bx = box + (size_t)leaf * 6;
  double acc[MAXC / FT];
  for (int q = 0; q < MAXC / FT; ++q) acc[q] = 0.0;
  for (int i0 = nb[leaf]; i0 < ne[leaf]; i0 += FT) {
    const int i = i0 + threadIdx.x;
    if (i < ne[leaf]) {
      for (int d = 0; d < D; ++d) {
        const double x = shift_coord(pos[(int64_t)d * npos + i], bx[d], bx[3 + d]);
        cheb_sn_tab(x, n, tab, &S[threadIdx.x][d * MAXN]);
      }
      sb[threadIdx.x] = b[i];
    }
    __syncthreads();
    const int cnt = min(FT, ne[leaf] - i0);
    for (int q = 0; q < MAXC / FT; ++q) {
      const int j = threadIdx.x + q * FT;
      if (j >= ncheb) break;
      double a = 0.0;
      for (int p = 0; p < cnt; ++p) {
        double r = sb[p];
        for (int d = 0; d < D; ++d) r *= S[p][d * MAXN + mi[j * 3 + d]];
        a += r;
      }
      acc[q] += a;
    }
    __syncthreads();
  }
  for (int q = 0; q < MAXC / FT; ++q) {
    const int j = threadIdx.x + q * FT;
    if (j < ncheb) W[(size_t)leaf * ncheb + j] = acc[q];
  }
}

// Mixed-precision P2M: the same sums in FP32 from the leaf-relative FP32
// positions (x = offset / half-width) and FP32 weights; each chunk of FT
// points is summed in FP32 and chunks are added in FP64.
__global__ void __launch_bounds__(FT) k_p2m32(int D, int n, int ncheb, const int *__restrict__ leaves,
                                              const int *__restrict__ nb, const int *__restrict__ ne,
                                              const double *__restrict__ box,
                                              const float4 *__restrict__ posf,
                                              const float *__restrict__ b32,
                                              const int *__restrict__ mi, const ChebTab32 tab,
                                              double *__restrict__ W) {
  __shared__ float S[FT][MAXN * 3 + 1];
  __shared__ float sb[FT];
  __shared__ int smi[MAXC * 3];
  const int leaf = leaves[blockIdx.x];
  const double *bx = box + (size_t)leaf * 6;
  float ihw[3] = {0.f, 0.f, 0.f};
  for (int d = 0; d < D; ++d) {
    const double hw = 0.5 * (bx[3 + d] - bx[d]);
    ihw[d] = hw > 0.0 ? (float)(1.0 / hw) : 0.f;
  }
  for (int e = threadIdx.x; e < ncheb * 3; e += FT) smi[e] = mi[e];
  double acc[MAXC / FT];
  for (int q = 0; q < MAXC / FT; ++q) acc[q] = 0.0;
  for (int i0 = nb[leaf]; i0 < ne[leaf]; i0 += FT) {
    const int i = i0 + threadIdx.x;
    if (i < ne[leaf]) {
      const float4 t = posf[i];
      const float xr[3] = {t.x, t.y, t.z};
      for (int d = 0; d < D; ++d) cheb_sn_tab32(xr[d] * ihw[d], n, tab, &S[threadIdx.x][d * MAXN]);
      sb[threadIdx.x] = b32[i];
    }
    __syncthreads();
    const int cnt = min(FT, ne[leaf] - i0);
    for (int q = 0; q < MAXC / FT; ++q) {
      const int j = threadIdx.x + q * FT;
      if (j >= ncheb) break;
      const int m0 = smi[j * 3], m1 = MAXN + smi[j * 3 + 1], m2 = 2 * MAXN + smi[j * 3 + 2];
      float a = 0.f;
      if (D == 3) {
        for (int p = 0; p < cnt; ++p) a = fmaf(sb[p] * S[p][m0], S[p][m1] * S[p][m2], a);
      } else {
        for (int p = 0; p < cnt; ++p) {
          float r = sb[p];
          for (int d = 0; d < D; ++d) r *= S[p][d * MAXN + smi[j * 3 + d]];
          a += r;
        }
      }
      acc[q] += (double)a;
    }
    __syncthreads();
  }
  for (int q = 0; q < MAXC / FT; ++q) {
    const int j = threadIdx.x + q * FT;
    if (j < ncheb) W[(size_t)leaf * ncheb + j] = acc[q];
  }
}

// ------------------------------------------------------------ M2M / L2L ---
// links: (parent, child, octant), sorted by octant within each level; one CTA
// per (batch of <= NBL links of one level and one octant, FT rows i), so
// that the CTA reads its rows of the octant's ncheb x ncheb matrix once for
// all the batch's links.
// M2M: W[p][i] += sum_j Tc[o][i][j] W[c][j]   (atomic over the parent's
//      children, which other batches hold); read through TcT[o][j][i] =
//      Tc[o][i][j] so that the loads are coalesced along i.
// L2L: G[c][i] += sum_j Tc[o][j][i] G[p][j]   (each child once).
// T is the compute type: double in FP64 mode; float in mixed mode (FP32
// copies of the matrices, FP32 sums of ncheb terms, FP64 storage).
// JS threads a row share its ncheb terms, and a term's NBL inputs are vector
// reads.  A row's walk of 343 loads from L2 is what a level with few links takes:
// four threads a row there; with links enough the shared sums only cost
// (launch_links has both sides).
constexpr int NBL = 8;  // links per M2M / L2L batch
template <typename T, bool M2M, int JS>
__global__ void __launch_bounds__(FT * JS) k_m2m_l2l(int ncheb, const int *__restrict__ links,
                                                     const int2 *__restrict__ batches,
                                                     const T *__restrict__ Tm_all,
                                                     double *__restrict__ V) {
  const int2 bt = batches[blockIdx.x];
  // inputs [j][link]; then the partial sums of all threads of a row but the first
  __shared__ __align__(16) T vin[MAXC][NBL];
  static_assert(MAXC >= (JS - 1) * FT, "the partial sums fit into the inputs' place");
  __shared__ int sout[NBL];
  const int o = links[3 * bt.x + 2];
  // M2M reads the children and writes the parents; L2L the other way round
  for (int e = threadIdx.x; e < NBL * ncheb; e += FT * JS) {
    const int b = e / ncheb, j = e - b * ncheb;
    T v = 0;
    if (b < bt.y) {
      const int nd = links[3 * (bt.x + b) + (M2M ? 1 : 0)];
      v = (T)V[(size_t)nd * ncheb + j];
    }
    vin[j][b] = v;
  }
  if (threadIdx.x < bt.y) sout[threadIdx.x] = links[3 * (bt.x + threadIdx.x) + (M2M ? 0 : 1)];
  __syncthreads();
  const T *Tm = Tm_all + (size_t)o * ncheb * ncheb;  // [j][i]
  const int it = threadIdx.x % FT, js = threadIdx.x / FT, i = blockIdx.y * FT + it;
  T a[NBL];
#pragma unroll
  for (int b = 0; b < NBL; ++b) a[b] = 0;
  if (i < ncheb) {
#pragma unroll 8
    for (int j = js; j < ncheb; j += JS) {
      const T t = Tm[(size_t)j * ncheb + i];
      T in[NBL];
      constexpr int V16 = 16 / sizeof(T);
#pragma unroll
      for (int q = 0; q < NBL / V16; ++q)
        *reinterpret_cast<int4 *>(&in[q * V16]) = *reinterpret_cast<const int4 *>(&vin[j][q * V16]);
#pragma unroll
      for (int b = 0; b < NBL; ++b) a[b] += t * in[b];
    }
  }
  __syncthreads();
  T(*part)[NBL] = vin;
  if (JS > 1 && js > 0)
#pragma unroll
    for (int b = 0; b < NBL; ++b) part[(js - 1) * FT + it][b] = a[b];
  __syncthreads();
  if (js > 0 || i >= ncheb) return;
  for (int q = 0; q < JS - 1; ++q)
#pragma unroll
    for (int b = 0; b < NBL; ++b) a[b] += part[q * FT + it][b];
#pragma unroll
  for (int b = 0; b < NBL; ++b) {
    if (b >= bt.y) break;
    double *dst = &V[(size_t)sout[b] * ncheb + i];
    if (M2M) atomicAdd(dst, (double)a[b]);
    else *dst += (double)a[b];
  }
}

// out[o][j][i] = (To)in[o][i][j] (transposed copy of the child matrices).
template <typename To>
__global__ void k_transpose_tc(const double *__restrict__ in, int nchild, int ncheb,
                               To *__restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)nchild * ncheb * ncheb) return;
  const int64_t o = e / ((int64_t)ncheb * ncheb);
  const int r = (int)(e % ((int64_t)ncheb * ncheb));
  const int j = r / ncheb, i = r % ncheb;
  out[e] = (To)in[(o * ncheb + i) * ncheb + j];
}

// --------------------------------------------------------------- M2L ---
// FP64 M2L as products of matrices of scaled 56-bit integers on the tensor cores
// (digits.cuh): for one matrix K and a tile of TC (target, source) pairs sharing
// it, TR rows of K W[:, sources], a warp 16 x 16 of them.  Digits are made once, of
// K per plan with a scale per row (Kd), of W per product with a scale per node
// (Wd).  A term is good to 2^-56 of the largest K of its row times the largest W of its
// node, so matrices with a row that spans more than fx::ONE_SIZE powers of two (a
// broad Gaussian's on coarse levels) are left to k_m2l64: their small entries would
// have fewer than FP64's 53 bits.  1 / d and sqrt(d^2 + c) stay within two at box
// distances of 1 to 2.45.  32 terms are staged at a time, the next while the last are
// multiplied.
// With FP64 one CTA a pair was bound by the pipe's 1.8 multiply-adds a clock and
// SM, with three 32x32+64-bit ones by their 25.  N = 1,048,576, 6.0e6 pairs: order 3
// (27 nodes) 8.5 -> 2.3 -> 1.8 ms; 100,000 points, order 5 (125), the whole
// product 20.8 -> 5.7 -> 3.6 ms.
using dg::MD;
constexpr int MF_K = 32;                // terms staged at a time
constexpr int MF_ROW = MD * MF_K;       // FP16 values of a row's 32 terms: [digit][term]
constexpr int MF_T = 256;
constexpr int mf_pairs(int nc) { return nc <= 32 ? 64 : 32; }  // pairs per tile
// Digits of `rows` rows of nc values, a warp a row; row r's 32 terms c go to
// ((r / per * chunks + c) * per + r % per) * MF_ROW (rows of one matrix together).
__global__ void __launch_bounds__(256) k_split_digits(const double *__restrict__ V, int64_t rows,
                                                      int nc, int per, __half *__restrict__ out,
                                                      short *__restrict__ exps) {
  const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const double *v = V + row * nc;
  fx::u64 mx = 0;
  for (int j = lane; j < nc; j += 32) mx = max(mx, fx::abs_bits(v[j]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int e = fx::scale_exp(mx), chunks = (nc + MF_K - 1) / MF_K;
  if (lane == 0) exps[row] = (short)e;
  for (int c = 0; c < chunks; ++c) {
    const int j = c * MF_K + lane;
    fx::i64 q = j < nc ? fx::whole56(v[j], e) : 0;
    __half *o = out + (((row / per) * chunks + c) * per + row % per) * MF_ROW + lane;
#pragma unroll
    for (int d = 0; d < MD; ++d) o[d * MF_K] = __low2half(dg::pair(fx::next_digit(q, d), 0));
  }
}

// Powers of two that the rows of each matrix span at most (fx::size_span): a CTA a
// matrix.
__global__ void __launch_bounds__(MF_T) k_row_span(const double *__restrict__ Km, int nc,
                                                   int *__restrict__ span) {
  __shared__ int most;
  if (threadIdx.x == 0) most = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < nc; i += MF_T / 32) {
    const double *row = Km + ((size_t)blockIdx.x * nc + i) * nc;
    int lo = 2047, hi = 0;
    for (int j = lane; j < nc; j += 32) {
      const int e = fx::size_of(row[j]);
      lo = min(lo, e);
      hi = max(hi, e);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) atomicMax(&most, fx::size_span(lo, hi));
  }
  __syncthreads();
  if (threadIdx.x == 0) span[blockIdx.x] = most;
}

// The same product in FP64, tiles of `pairs` pairs of one matrix a CTA, four of them
// with every K that is read.  Bound by the FP64 pipe.
constexpr int MW_PAIRS = 16;  // (P->tile_mat, whatever its tiles, does as well)
__global__ void __launch_bounds__(FT) k_m2l64(int ncheb, const double *__restrict__ Km,
                                              const int2 *__restrict__ by_mat,
                                              const int *__restrict__ mat_off,
                                              const int *__restrict__ tile_mat,
                                              const int *__restrict__ tile_first, int pairs,
                                              const double *__restrict__ W,
                                              double *__restrict__ G) {
  constexpr int U = 4;
  __shared__ double ws[MAXC][U];
  const int m = tile_mat[blockIdx.x], first = tile_first[blockIdx.x];
  const int last = min(first + pairs, mat_off[m + 1]);
  const double *K = Km + (size_t)m * ncheb * ncheb;
  for (int q = first; q < last; q += U) {
    const int np = min(U, last - q);
    __syncthreads();
    for (int e = threadIdx.x; e < U * ncheb; e += FT) {
      const int u = e / ncheb, j = e - u * ncheb;
      ws[j][u] = u < np ? W[(size_t)by_mat[q + u].y * ncheb + j] : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ncheb; i += FT) {
      double a[U] = {};
      for (int j = 0; j < ncheb; ++j) {
        const double k = K[(size_t)i * ncheb + j];
#pragma unroll
        for (int u = 0; u < U; ++u) a[u] += k * ws[j][u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < np) atomicAdd(&G[(size_t)by_mat[q + u].x * ncheb + i], a[u]);
    }
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// 16-byte asynchronous copy; nbytes = 0 writes zeros.
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, int nbytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(nbytes)
               : "memory");
}

// Byte offset of digit d, row r (of a tile's R), 16-byte chunk c of 4: permuted, so
// that ldmatrix reads 8 rows without conflicts.
template <int R> __device__ __forceinline__ uint32_t mf_at(int d, int r, int c) {
  return (uint32_t)((d * R + r) * 64 + ((c ^ ((r >> 1) & 3)) << 4));
}
template <int TR, int TC> constexpr size_t mf_stage() { return (size_t)MD * (TR + TC) * MF_K * 2; }

template <int TR, int TC, int STAGES>
__global__ void __launch_bounds__(MF_T, 2) k_m2l_fix(
    int nc, const __half *__restrict__ Kd, const short *__restrict__ ke,
    const __half *__restrict__ Wd, const short *__restrict__ we, const int2 *__restrict__ by_mat,
    const int *__restrict__ mat_off, const int *__restrict__ tile_mat,
    const int *__restrict__ tile_first, double *__restrict__ G) {
  static_assert((TR / 16) * (TC / 16) == MF_T / 32, "16 x 16 a warp");
  extern __shared__ __align__(128) unsigned char mf_raw[];
  __shared__ int tgt[TC], src[TC], sexp[TC];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = tile_mat[blockIdx.x], first = tile_first[blockIdx.x];
  const int np = min(TC, mat_off[m + 1] - first), r0 = blockIdx.y * TR;
  if (tid < TC) {
    const int2 ts = by_mat[first + min(tid, np - 1)];
    tgt[tid] = ts.x;
    src[tid] = ts.y;
    sexp[tid] = we[ts.y];
  }
  __syncthreads();
  const uint32_t base = smem_addr(mf_raw);
  const int chunks = (nc + MF_K - 1) / MF_K;
  const int wr = (warp % (TR / 16)) * 16, wc = (warp / (TR / 16)) * 16;
  auto load = [&](int c) {  // terms 32 c .. of the tile's rows and sources
    const uint32_t st = base + (uint32_t)((c % STAGES) * mf_stage<TR, TC>());
    constexpr int PIECES = MF_ROW * 2 / 16;
    for (int e = tid; e < (TR + TC) * PIECES; e += MF_T) {
      const int r = e / PIECES, q = e - r * PIECES, d = q >> 2, ch = q & 3;
      if (r < TR) {
        const bool in = r0 + r < nc;
        cp16(st + mf_at<TR>(d, r, ch),
             Kd + (((size_t)m * chunks + c) * nc + (in ? r0 + r : 0)) * MF_ROW + q * 8, in ? 16 : 0);
      } else {
        const int p = r - TR;
        cp16(st + (uint32_t)(MD * TR * MF_K * 2) + mf_at<TC>(d, p, ch),
             Wd + ((size_t)src[p] * chunks + c) * MF_ROW + q * 8, 16);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[MD][2][4] = {};
  double total[2][4] = {};
  load(0);
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    if (STAGES > 1 && c + 1 < chunks) {
      load(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const uint32_t sA = base + (uint32_t)((c % STAGES) * mf_stage<TR, TC>());
    const uint32_t sB = sA + (uint32_t)(MD * TR * MF_K * 2);
    if (r0 + wr < nc && wc < np) {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        if (c * MF_K + h * 16 >= nc) break;
        uint32_t a[MD][4];
#pragma unroll
        for (int d = 0; d < MD; ++d)
          dg::ldmatrix4(a[d], sA + mf_at<TR>(d, wr + (lane & 15), 2 * h + (lane >> 4)));
#pragma unroll
        for (int d = 0; d < MD; ++d) {
          uint32_t b[4];
          dg::ldmatrix4(b, sB + mf_at<TC>(d, wc + (lane & 7) + (lane >> 4) * 8, 2 * h + ((lane >> 3) & 1)));
          dg::multiply(acc, a, b, d);
        }
      }
      if (STAGES > 1 && ((c + 1) * MF_K % dg::MAX_TERMS == 0 || c + 1 == chunks)) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int q = 0; q < 4; ++q) total[b][q] += (double)dg::sum(acc, b, q);
#pragma unroll
        for (int w = 0; w < MD; ++w)
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[w][b][q] = 0.f;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + wr + (lane >> 2) + 8 * (q >> 1), p = wc + 8 * b + 2 * (lane & 3) + (q & 1);
      if (r >= nc || p >= np) continue;
      const double t = STAGES > 1 ? total[b][q] : (double)dg::sum(acc, b, q);
      atomicAdd(&G[(size_t)tgt[p] * nc + r], fx::times56(t, (int)ke[(size_t)m * nc + r] + sexp[p]));
    }
}

// Mixed precision M2L on the tensor cores: for one matrix K (ncheb x ncheb,
// FP32) and a tile of 64 (target, source) pairs sharing it:
//   C[16 x 64] (rows i0..i0+15) = K[i0:i0+16, :] * W[:, sources]
// as 3xTF32 (a = ah + al, b = bh + bl; ah*bh + ah*bl + al*bh) on
// mma.sync.m16n8k8.tf32 with FP32 accumulation, then atomically added to G.
__device__ __forceinline__ uint32_t f2tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mma_tf32(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int TC_PAIRS = 64;  // pairs per CTA

// Split-TF32 parts of the FP32 M2L matrices: hi = tf32(K), lo = tf32(K - hi),
// so that K ~= hi + lo to ~2^-22 and K W ~= hi Wh + hi Wl + lo Wh.
// Rows of ncheb entries are stored with stride ldk (a multiple of 32, zero
// padded), so that the tensor-core kernels stage whole 16-byte-aligned
// 32-column blocks.
__global__ void k_split_tf32(const double *__restrict__ K, int64_t nrows, int ncheb, int ldk,
                             float *__restrict__ hi, float *__restrict__ lo) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nrows * ldk) return;
  const int64_t row = e / ldk;
  const int k = (int)(e % ldk);
  const float f = k < ncheb ? (float)K[row * ncheb + k] : 0.f;
  const uint32_t h = f2tf32(f);
  hi[e] = __uint_as_float(h);
  lo[e] = __uint_as_float(f2tf32(f - __uint_as_float(h)));
}

// W32[node][k] = (float)W[node][k] with row stride ldk (zero padded).
__global__ void k_to_f32_padded(const double *__restrict__ W, int64_t nrows, int ncheb, int ldk,
                                float *__restrict__ W32) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nrows * ldk) return;
  const int64_t row = e / ldk;
  const int k = (int)(e % ldk);
  W32[e] = k < ncheb ? (float)W[row * ncheb + k] : 0.f;
}

// Tensor-core M2L, one CTA per (M2L matrix, 64-pair tile, MT-row block):
// G[tgt_q][rows] += K[rows][:] W[src_q][:] for the tile's pairs q, as an
// MT x 64 x ncheb GEMM in 3xTF32 (mma.sync m16n8k8, FP32 accumulation).
// WM x 2 warps (rows x pairs), 32 x 32 per warp, MT = 32 WM chosen from the
// number of Chebyshev nodes; K and W are staged 32 columns at a time in
// padded shared memory (conflict-free fragment loads); the accumulators
// leave through shared memory as 16-byte vector reductions into G (row
// stride ldg, a multiple of 4).
constexpr int M2_NT = 64, M2_KB = 32, M2_LD = M2_KB + 4;
template <int WM> struct M2Cfg {
  static constexpr int MT = 32 * WM, LDC = MT + 4, THREADS = 64 * WM;
  static constexpr size_t SMEM =
      (size_t)(2 * MT * M2_LD + 2 * M2_NT * M2_LD) * sizeof(float) + 2 * M2_NT * sizeof(int);
  static_assert((size_t)M2_NT * LDC <= (size_t)(2 * MT * M2_LD + 2 * M2_NT * M2_LD),
                "the epilogue tile reuses the staging area");
};

template <int WM>
__global__ void __launch_bounds__(64 * WM) k_m2l_tc2(int ncheb, int ldk, int ldg, const float *__restrict__ Kh,
                                                 const float *__restrict__ Kl,
                                                 const int2 *__restrict__ pairs,
                                                 const int *__restrict__ mat_off,
                                                 const int *__restrict__ tile_mat,
                                                 const int *__restrict__ tile_first,
                                                 const float *__restrict__ W32,
                                                 float *__restrict__ G32) {
  constexpr int M2_MT = M2Cfg<WM>::MT, M2_LDC = M2Cfg<WM>::LDC, NTH = M2Cfg<WM>::THREADS;
  extern __shared__ __align__(16) float m2s[];
  float *sAh = m2s, *sAl = sAh + M2_MT * M2_LD;
  float *sBh = sAl + M2_MT * M2_LD, *sBl = sBh + M2_NT * M2_LD;
  int *sSrc = (int *)(sBl + M2_NT * M2_LD), *sTgt = sSrc + M2_NT;
  float *sC = m2s;  // epilogue, after the main loop
  const int tile = blockIdx.x, i0 = blockIdx.y * M2_MT;
  const int m = tile_mat[tile], p0 = tile_first[tile];
  const int np = min(M2_NT, mat_off[m + 1] - p0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = warp % WM, wn = warp / WM;
  if (tid < M2_NT) {
    const int2 pr = tid < np ? pairs[p0 + tid] : make_int2(-1, -1);
    sTgt[tid] = pr.x;
    sSrc[tid] = pr.y;
  }
  const float *Ah = Kh + (size_t)m * ncheb * ldk, *Al = Kl + (size_t)m * ncheb * ldk;
  float c[2][4][4] = {};
  for (int k0 = 0; k0 < ncheb; k0 += M2_KB) {
    __syncthreads();
    for (int e = tid; e < M2_MT * M2_KB; e += NTH) {
      const int r = e / M2_KB, cc = e % M2_KB, i = i0 + r, k = k0 + cc;
      const bool in = i < ncheb && k < ncheb;
      sAh[r * M2_LD + cc] = in ? Ah[(size_t)i * ldk + k] : 0.f;
      sAl[r * M2_LD + cc] = in ? Al[(size_t)i * ldk + k] : 0.f;
    }
    for (int e = tid; e < M2_NT * M2_KB; e += NTH) {
      const int q = e / M2_KB, cc = e % M2_KB, k = k0 + cc;
      const int sidx = sSrc[q];
      const float v = (sidx >= 0 && k < ncheb) ? W32[(size_t)sidx * ldk + k] : 0.f;
      const uint32_t h = f2tf32(v);
      sBh[q * M2_LD + cc] = __uint_as_float(h);
      sBl[q * M2_LD + cc] = __uint_as_float(f2tf32(v - __uint_as_float(h)));
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < M2_KB; kk += 8) {
      uint32_t ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
      for (int mf = 0; mf < 2; ++mf) {
        const int r = wm * 32 + mf * 16 + g;
        ah[mf][0] = __float_as_uint(sAh[r * M2_LD + kk + t4]);
        ah[mf][1] = __float_as_uint(sAh[(r + 8) * M2_LD + kk + t4]);
        ah[mf][2] = __float_as_uint(sAh[r * M2_LD + kk + t4 + 4]);
        ah[mf][3] = __float_as_uint(sAh[(r + 8) * M2_LD + kk + t4 + 4]);
        al[mf][0] = __float_as_uint(sAl[r * M2_LD + kk + t4]);
        al[mf][1] = __float_as_uint(sAl[(r + 8) * M2_LD + kk + t4]);
        al[mf][2] = __float_as_uint(sAl[r * M2_LD + kk + t4 + 4]);
        al[mf][3] = __float_as_uint(sAl[(r + 8) * M2_LD + kk + t4 + 4]);
      }
#pragma unroll
      for (int nf = 0; nf < 4; ++nf) {
        const int q = wn * 32 + nf * 8 + g;
        bh[nf][0] = __float_as_uint(sBh[q * M2_LD + kk + t4]);
        bh[nf][1] = __float_as_uint(sBh[q * M2_LD + kk + t4 + 4]);
        bl[nf][0] = __float_as_uint(sBl[q * M2_LD + kk + t4]);
        bl[nf][1] = __float_as_uint(sBl[q * M2_LD + kk + t4 + 4]);
      }
#pragma unroll
      for (int mf = 0; mf < 2; ++mf)
#pragma unroll
        for (int nf = 0; nf < 4; ++nf) {
          mma_tf32(c[mf][nf], al[mf], bh[nf]);
          mma_tf32(c[mf][nf], ah[mf], bl[nf]);
          mma_tf32(c[mf][nf], ah[mf], bh[nf]);
        }
    }
  }
  __syncthreads();
  // C fragments -> sC[pair][row]
#pragma unroll
  for (int mf = 0; mf < 2; ++mf)
#pragma unroll
    for (int nf = 0; nf < 4; ++nf) {
      const int r = wm * 32 + mf * 16 + g, q = wn * 32 + nf * 8 + 2 * t4;
      sC[q * M2_LDC + r] = c[mf][nf][0];
      sC[(q + 1) * M2_LDC + r] = c[mf][nf][1];
      sC[q * M2_LDC + r + 8] = c[mf][nf][2];
      sC[(q + 1) * M2_LDC + r + 8] = c[mf][nf][3];
    }
  __syncthreads();
  for (int e = tid; e < M2_NT * (M2_MT / 4); e += NTH) {
    const int q = e / (M2_MT / 4), r4 = (e % (M2_MT / 4)) * 4;
    const int tgt = sTgt[q];
    if (tgt < 0 || i0 + r4 >= ncheb) continue;
    const float4 v = *reinterpret_cast<const float4 *>(&sC[q * M2_LDC + r4]);
    float *dst = G32 + (size_t)tgt * ldg + i0 + r4;  // 16-byte aligned: ldg, i0 + r4 multiples of 4
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y),
                 "f"(v.z), "f"(v.w)
                 : "memory");
  }
}

// ------------------------------------------------- M2L on tcgen05 (TMEM) ---
// The same tile GEMM on the 5th-generation tensor cores.  One CTA (4 warps)
// per (M2L matrix, N-pair tile) computes all NRB = ceil(ncheb/128) row
// blocks, so the gathered source expansions of the tile are read once:
//   G[targets][rb*128 + r] += sum_k K[rb*128 + r][k] * W[sources][k]
// as split FP16 (K = Kh + Kl, W = Wh + Wl; Kl Wh + Kh Wl + Kh Wh) on
// tcgen05.mma kind::f16 into NRB accumulators of 128 x N FP32 in TMEM.  Every K
// matrix and every node's W has its own power of two, which brings its largest
// value to [2^14, 2^15): hi and lo then have the 11 + 11 bits that TF32 parts
// have for entries down to 2^-17 of the largest, and all entries are good to 2^-39
// of it, far below the 2^-24 to which the FP32 W are.  Against FP64 sums of 20,000
// points (1 / (d + c), multiquadric, Gaussians of p0 = 2, 30 and 200; weights of one
// sign, of two, over 2^40; orders 5 and 7) no product's error in norm was larger
// than with split TF32, the smallest was 0.3 of it.  A 16-byte chunk, a stage and an
// MMA hold twice the columns; the tensor pipe's FP16 rate is twice TF32's, and the
// operands' shared-memory traffic, which bounds 64-pair tiles, is half.  Order 7,
// N = 1M: 10.4 -> 6.2 ms (the loads and the reductions into G alone, without an MMA,
// take 6.5).
// The K matrices are packed once per plan into the shared-memory image of a
// pipeline stage (k_pack_f16), so a stage's A operand is one bulk copy on the
// TMA engine (cp.async.bulk, completion counted on the stage's `fullA`
// mbarrier) and bypasses the load/store pipeline; the W rows of the tile's
// sources are gathered 16 bytes per lane with cp.async.  Operands use the
// no-swizzle K-major core-matrix layout (8 rows x 16 bytes per core matrix;
// the descriptor's leading byte offset is the core-matrix stride along K, the
// stride byte offset along rows).
// Roles, with no CTA-wide barrier inside the loop: warp 0 produces (waits for
// the stage's `empty` barrier, issues block p, then waits for block p-LAG's
// W copies, fences them to the async proxy and arrives on `fullB`); lane 0 of
// warp 1 waits for `fullA` and `fullB`, issues the 3 NRB MMAs of the block
// and commits them to `empty`, and after the last block to `accb`; all four
// warps then wait for `accb` and run the epilogue: each reads its 32
// accumulator lanes (rows) with tcgen05.ld and adds them into G with
// reductions that are coalesced along the rows.  Every wait is bounded: on
// timeout the kernel sets *status, skips the epilogue, waits (bounded) for
// its copies and MMAs in flight and still releases its TMEM.  The ring depth
// keeps the CTAs resident on an SM (by shared memory) within the SM's 512
// TMEM columns.
constexpr int T5_KB = 16;
constexpr int T5_PART = 128 * T5_KB * 2;  // bytes of one K operand part: 128 rows x 16 columns
constexpr uint32_t T5_POLL_CAP = 1u << 30;  // second bound on the polls of one wait
// Per row-block count: N pairs per tile, ring depth S, producer lag LAG and
// TMEM columns.  Three or four row blocks use 64-pair tiles so that two CTAs
// share an SM (their latencies overlap); one or two use 128-pair tiles.
template <int NRB> struct T5Cfg {
  static constexpr int N = NRB <= 2 ? 128 : 64;
  static constexpr int S = NRB == 2 ? 4 : 3;  // ring depth
  // the producer signals block p - LAG's W copies after issuing block p
  // (LAG < S: the MMAs of block p - S, which free block p's stage, never wait
  // for a block the producer has not signalled)
  static constexpr int LAG = NRB == 2 ? 2 : 1;
  static constexpr int A_BYTES = NRB * 2 * T5_PART;       // K hi, lo of every row block
  static constexpr int B_PART = N * T5_KB * 2;            // W of the N pairs, one part
  static constexpr int STAGE = A_BYTES + 2 * B_PART;
  static constexpr size_t SMEM = (size_t)S * STAGE + 1024 + 2048;  // + alignment, barriers, indices
  static constexpr uint32_t TCOLS = NRB * N <= 128 ? 128u : (NRB * N <= 256 ? 256u : 512u);
};
constexpr int t5_pairs(int nrb) { return nrb <= 2 ? T5Cfg<1>::N : T5Cfg<3>::N; }
static_assert(T5Cfg<1>::N == T5Cfg<2>::N && T5Cfg<3>::N == T5Cfg<4>::N, "tile width per t5_pairs");
// resident CTAs per SM (bounded by shared memory) x TCOLS <= the SM's 512 TMEM columns
static_assert(T5Cfg<1>::SMEM * 5 > 228 * 1024 && T5Cfg<2>::SMEM * 3 > 228 * 1024 &&
                  T5Cfg<3>::SMEM * 3 > 228 * 1024 && T5Cfg<4>::SMEM * 3 > 228 * 1024,
              "resident CTAs per SM must fit the SM's 512 TMEM columns");
static_assert(T5Cfg<3>::SMEM <= 227 * 1024 && T5Cfg<4>::SMEM <= 227 * 1024, "shared memory per CTA");
static_assert(T5Cfg<1>::LAG < T5Cfg<1>::S && T5Cfg<2>::LAG < T5Cfg<2>::S &&
                  T5Cfg<3>::LAG < T5Cfg<3>::S && T5Cfg<4>::LAG < T5Cfg<4>::S,
              "producer lag below the ring depth");

// Power of two that brings values up to `big` to [2^14, 2^15) (in FP32's range;
// 1 for zero), as the factor that takes them back.
__device__ __forceinline__ float f16_unit(float big) {
  if (!(big > 0.f && big <= 3.4e38f)) return 1.f;
  int e;
  frexpf(big, &e);
  return ldexpf(1.f, min(max(e - 15, -126), 113));
}

// Power of two of each M2L matrix: a CTA a matrix.
constexpr int KS_TPB = 256;
__global__ void __launch_bounds__(KS_TPB) k_mat_scale(const double *__restrict__ K, int64_t len,
                                                      float *__restrict__ scale) {
  __shared__ float part[KS_TPB / 32];
  float big = 0.f;
  for (int64_t i = threadIdx.x; i < len; i += KS_TPB)
    big = fmaxf(big, fabsf((float)K[blockIdx.x * len + i]));
  for (int d = 16; d > 0; d >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, d));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = big;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < KS_TPB / 32; ++w) big = fmaxf(big, part[w]);
    scale[blockIdx.x] = f16_unit(big);
  }
}

// Packed split-FP16 M2L matrices: per (matrix, 16-column block kb, 128-row
// block rb, part hi/lo) the 4 KB shared-memory image of the operand tile,
// element (r, k) at ((k/8) * 16 + r/8) * 128 + (r%8) * 16 + (k%8) * 2 bytes;
// zero beyond ncheb.  hi = fp16(K / scale), lo = fp16(K / scale - hi).
__global__ void k_pack_f16(const double *__restrict__ K, const float *__restrict__ scale,
                           int64_t nmat, int ncheb, int nkb, int nrb, __half *__restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nmat * nkb * nrb * 2 * (T5_PART / 2)) return;
  int64_t t = e;
  const int w = (int)(t % (T5_PART / 2));
  t /= T5_PART / 2;
  const int part = (int)(t % 2);
  t /= 2;
  const int rb = (int)(t % nrb);
  t /= nrb;
  const int kb = (int)(t % nkb);
  const int64_t m = t / nkb;
  const int kk = w & 7, rl = (w >> 3) & 7, rh = (w >> 6) & 15, kq = w >> 10;
  const int i = rb * 128 + rh * 8 + rl, k = kb * T5_KB + kq * 8 + kk;
  // (scale: a power of two down to 2^-126, whose reciprocal is a float)
  const float f =
      (i < ncheb && k < ncheb) ? (float)K[(m * ncheb + i) * ncheb + k] * (1.f / scale[m]) : 0.f;
  const __half h = __float2half_rn(f);
  out[e] = part == 0 ? h : __float2half_rn(f - __half2float(h));
}

// W as scaled split FP16 (rows of ldk values, zero beyond ncheb): a warp a node.
__global__ void __launch_bounds__(256) k_split_f16(const double *__restrict__ W, int64_t nnodes,
                                                   int ncheb, int ldk, __half *__restrict__ hi,
                                                   __half *__restrict__ lo,
                                                   float *__restrict__ scale) {
  const int64_t node = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (node >= nnodes) return;
  float v[16];  // ncheb <= 512
  float big = 0.f;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int k = q * 32 + lane;
    v[q] = k < ncheb ? (float)W[node * ncheb + k] : 0.f;
    big = fmaxf(big, fabsf(v[q]));
  }
  for (int d = 16; d > 0; d >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, d));
  const float unit = f16_unit(big), inv = 1.f / unit;
  if (lane == 0) scale[node] = unit;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int k = q * 32 + lane;
    if (k >= ldk) break;
    const float f = v[q] * inv;
    const __half h = __float2half_rn(f);
    hi[node * ldk + k] = h;
    lo[node * ldk + k] = __float2half_rn(f - __half2float(h));
  }
}

// Shared-memory matrix descriptor: no swizzle, K-major.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor, kind::f16: D F32, A and B FP16, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Wait for the given phase of an mbarrier for at most limit_ns nanoseconds
// of the GPU's global timer (and at most T5_POLL_CAP polls); false if it ran
// out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t it = 0; it < T5_POLL_CAP; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 15u) == 0u) {
      const uint64_t now = globaltimer_ns();
      if (it == 0u)
        t0 = now;
      else if (now - t0 > limit_ns)
        return false;
    }
  }
  return false;
}

template <int NRB>
__global__ void __launch_bounds__(128) k_m2l_tc5(int ncheb, int nkb, int ldk, int ldg,
                                                 const __half *__restrict__ Ap,
                                                 const float *__restrict__ Ap_scale,
                                                 const int2 *__restrict__ pairs,
                                                 const int *__restrict__ mat_off,
                                                 const int *__restrict__ tile_mat,
                                                 const int *__restrict__ tile_first,
                                                 const __half *__restrict__ Wh,
                                                 const __half *__restrict__ Wl,
                                                 const float *__restrict__ W_scale,
                                                 float *__restrict__ G32, int *__restrict__ status,
                                                 uint64_t limit_ns, int drop_arrive) {
  using C = T5Cfg<NRB>;
  constexpr int S = C::S, LAG = C::LAG, T5_N = C::N;
  extern __shared__ __align__(128) unsigned char t5raw[];
  unsigned char *sm = (unsigned char *)(((uintptr_t)t5raw + 1023) & ~(uintptr_t)1023);
  uint64_t *fullA = (uint64_t *)(sm + S * C::STAGE);
  uint64_t *fullB = fullA + S, *empty = fullB + S, *accb = empty + S;
  uint32_t *tslot = (uint32_t *)(accb + 1);
  int *sSrc = (int *)(tslot + 4), *sTgt = sSrc + T5_N, *sInfo = sTgt + T5_N;
  float *sScale = (float *)(sInfo + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x;
  const int m = tile_mat[tile], p0 = tile_first[tile];
  const int np = min(T5_N, mat_off[m + 1] - p0);
  if (tid < T5_N) {
    const int2 pr = tid < np ? pairs[p0 + tid] : make_int2(-1, -1);
    sTgt[tid] = pr.x;
    sSrc[tid] = pr.y;
    sScale[tid] = pr.y >= 0 ? W_scale[pr.y] : 0.f;
  }
  const float mat_scale = Ap_scale[m];
  if (tid == 0) {
    for (int q = 0; q < S; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&fullA[q])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&fullB[q])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&empty[q])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(accb)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sInfo[0] = 0;  // blocks issued by the producer
    sInfo[1] = 0;  // blocks whose operands the MMA issuer received
    sInfo[2] = 1;  // producer ok
    sInfo[3] = 1;  // MMA issuer ok
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tslot)),
                 "r"(C::TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t smbase = smem_addr(sm);

  if (warp == 0) {
    // ---- producer
    const unsigned char *Am = (const unsigned char *)Ap + (size_t)m * nkb * C::A_BYTES;
    bool ok = true;
    int p = 0;
    for (; p < nkb; ++p) {
      const int st = p % S;
      if (p >= S && !mbar_wait(smem_addr(&empty[st]), ((p - S) / S) & 1, limit_ns)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint32_t sb = smbase + (uint32_t)(st * C::STAGE);
      if (lane == 0) {
        const uint32_t fb = smem_addr(&fullA[st]);
        asm volatile(
            "{\n\t.reg .b64 state;\n\t"
            "mbarrier.arrive.expect_tx.shared::cta.b64 state, [%0], %1;\n\t}" ::"r"(fb),
            "r"(C::A_BYTES)
            : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(sb),
            "l"(Am + (size_t)p * C::A_BYTES), "r"(C::A_BYTES), "r"(fb)
            : "memory");
      }
#pragma unroll
      for (int e = lane; e < T5_N * (T5_KB / 8); e += 32) {
        const int rl = e & 7, kq = (e >> 3) & 1, rh = e >> 4;
        const int src = sSrc[rh * 8 + rl];
        const uint32_t off = (uint32_t)((kq * (T5_N / 8) + rh) * 128 + rl * 16);
        const size_t g = (size_t)(src >= 0 ? src : 0) * ldk + p * T5_KB + kq * 8;
        cp16(sb + C::A_BYTES + off, Wh + g, src >= 0 ? 16 : 0);
        cp16(sb + C::A_BYTES + C::B_PART + off, Wl + g, src >= 0 ? 16 : 0);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (p >= LAG) {
        // block p - LAG's W copies have landed: hand them to the async proxy
        asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        // drop_arrive (fault injection for tests): block 0's W copies are
        // never signalled, so the MMA issuer's wait runs out
        if (lane == 0 && !(drop_arrive && p - LAG == 0))
          asm volatile("{\n\t.reg .b64 state;\n\tmbarrier.arrive.shared::cta.b64 state, [%0];\n\t}" ::"r"(
                           smem_addr(&fullB[(p - LAG) % S]))
                       : "memory");
      }
    }
    // the last min(p, LAG) blocks
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      for (int q = max(p - LAG, 0); q < p; ++q)
        if (!(drop_arrive && q == 0))
          asm volatile("{\n\t.reg .b64 state;\n\tmbarrier.arrive.shared::cta.b64 state, [%0];\n\t}" ::"r"(
                         smem_addr(&fullB[q % S]))
                     : "memory");
      sInfo[0] = p;
      if (!ok) sInfo[2] = 0;
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    constexpr uint32_t idesc = umma_idesc_f16(128, T5_N);
    constexpr uint32_t ks = (128 / 8) * 128;    // core-matrix stride along K (K rows)
    constexpr uint32_t bks = (T5_N / 8) * 128;  // the same for the T5_N pair rows
    bool ok = true;
    int c = 0;
    for (; c < nkb; ++c) {
      const int st = c % S;
      const uint32_t par = (c / S) & 1;
      if (!mbar_wait(smem_addr(&fullA[st]), par, limit_ns) ||
          !mbar_wait(smem_addr(&fullB[st]), par, limit_ns)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t base = smbase + (uint32_t)(st * C::STAGE);
      const uint64_t bh = umma_desc(base + C::A_BYTES, bks, 128);
      const uint64_t bl = umma_desc(base + C::A_BYTES + C::B_PART, bks, 128);
#pragma unroll
      for (int rb = 0; rb < NRB; ++rb) {
        const uint64_t ah = umma_desc(base + rb * 2 * T5_PART, ks, 128);
        const uint64_t al = umma_desc(base + rb * 2 * T5_PART + T5_PART, ks, 128);
        const uint64_t ad[3] = {al, ah, ah}, bd[3] = {bh, bl, bh};
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const uint32_t acc = (c > 0 || t > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
                  tmem + (uint32_t)(rb * T5_N)),
              "l"(ad[t]), "l"(bd[t]), "r"(idesc), "r"(acc));
        }
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_addr(&empty[st])));
    }
    // completes once every MMA issued above has completed
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_addr(accb)));
    sInfo[1] = c;
    if (!ok) sInfo[3] = 0;
  }
  __syncthreads();
  const bool acc_ready = mbar_wait(smem_addr(accb), 0, limit_ns);
  const bool ok = __syncthreads_and(acc_ready && sInfo[2] && sInfo[3] && sInfo[1] == nkb);
  if (!ok) {
    if (tid == 0) {
      atomicExch(status, 1);
      // the MMAs issued so far (accb) and the bulk copies still in flight
      // (fullA) complete before TMEM and shared memory are released; each of
      // these waits is bounded as well
      if (!acc_ready) mbar_wait(smem_addr(accb), 0, limit_ns);
      for (int q = sInfo[1]; q < sInfo[0]; ++q)
        mbar_wait(smem_addr(&fullA[q % S]), (q / S) & 1, limit_ns);
    }
    __syncthreads();
  } else {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // per warp a 16 x 32 transpose tile in the (now idle) first stage: lane
    // = row on the way in, (pair, 4 consecutive rows) on the way out, so that
    // G receives 16-byte vector reductions (ldg and the row groups are
    // multiples of 4; groups at or beyond ncheb are skipped)
    float *tt = reinterpret_cast<float *>(sm) + warp * (16 * 32);
#pragma unroll 1
    for (int rb = 0; rb < NRB; ++rb) {
      const int i0 = rb * 128 + 32 * warp;
#pragma unroll 1
      for (int c0 = 0; c0 < T5_N; c0 += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(rb * T5_N + c0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 16; ++q) tt[q * 32 + lane] = __uint_as_float(v[q]);
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int q = it * 4 + (lane >> 3), g = (lane & 7) * 4;
          const int tgt = sTgt[c0 + q];
          if (tgt >= 0 && i0 + g < ncheb) {
            const float4 a = *reinterpret_cast<const float4 *>(&tt[q * 32 + g]);
            const float sc = sScale[c0 + q];
            float *dst = G32 + (size_t)tgt * ldg + i0 + g;
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst),
                         "f"(a.x * mat_scale * sc), "f"(a.y * mat_scale * sc),
                         "f"(a.z * mat_scale * sc), "f"(a.w * mat_scale * sc)
                         : "memory");
          }
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TCOLS));
}

// G[node][i] += G32[node][i] for the padded FP32 accumulator (row stride ldg).
__global__ void k_add_g32(const float *__restrict__ G32, int64_t nnodes, int ncheb, int ldg,
                          double *__restrict__ G) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nnodes * ncheb) return;
  const int64_t node = e / ncheb;
  const int i = (int)(e % ncheb);
  G[e] += (double)G32[node * ldg + i];
}

__global__ void k_f64_to_f32(const double *__restrict__ a, int64_t n, float *__restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

// ----------------------------------------------------------- L2P + P2P ---
template <int KIND, bool MIXED>
__global__ void __launch_bounds__(FT) k_l2p_p2p(int D, int n, int ncheb, const int *__restrict__ leaves,
                                                const int *__restrict__ nb,
                                                const int *__restrict__ ne,
                                                const double *__restrict__ box,
                                                const double *__restrict__ pos, int64_t npos,
                                                const double *__restrict__ b,
                                                const int *__restrict__ mi,
                                                const double *__restrict__ G,
                                                const int *__restrict__ rp,
                                                const int *__restrict__ src, double p0,
                                                const ChebTab tab, double *__restrict__ c) {
  __shared__ double sg[MAXC];
  __shared__ double sx[FT], sy[FT], sz[FT], sbv[FT];
  __shared__ int sid[FT];
  const int li = blockIdx.x;
  const int leaf = leaves[li];
  const double *bx = box + (size_t)leaf * 6;
  for (int j = threadIdx.x; j < ncheb; j += FT) sg[j] = G[(size_t)leaf * ncheb + j];
  __syncthreads();
  for (int i0 = nb[leaf]; i0 < ne[leaf]; i0 += FT) {
    const int i = i0 + threadIdx.x;
    const bool act = i < ne[leaf];
    double xi[3] = {0, 0, 0};
    double acc = 0.0;
    if (act) {
      for (int d = 0; d < D; ++d) xi[d] = pos[(int64_t)d * npos + i];
      double S[3][MAXN];
      for (int d = 0; d < D; ++d) cheb_sn_tab(shift_coord(xi[d], bx[d], bx[3 + d]), n, tab, S[d]);
      for (int j = 0; j < ncheb; ++j) {
        double r = sg[j];
        for (int d = 0; d < D; ++d) r *= S[d][mi[j * 3 + d]];
        acc += r;
      }
    }
    // P2P over the connected source leaves
    for (int e = rp[li]; e < rp[li + 1]; ++e) {
      const int sl = src[e];
      for (int j0 = nb[sl]; j0 < ne[sl]; j0 += FT) {
        __syncthreads();
        const int j = j0 + threadIdx.x;
        if (j < ne[sl]) {
          sx[threadIdx.x] = pos[j];
          sy[threadIdx.x] = D > 1 ? pos[npos + j] : 0.0;
          sz[threadIdx.x] = D > 2 ? pos[2 * npos + j] : 0.0;
          sbv[threadIdx.x] = b[j];
          sid[threadIdx.x] = j;
        }
        __syncthreads();
        const int cnt = min(FT, ne[sl] - j0);
        if (act) {
          if (MIXED) {
            // FP32 pair terms summed per staged chunk, chunks summed in FP64;
            // the self pair (a regularised singular kernel can be huge there)
            // is evaluated in FP64.
            float a = 0.f;
            for (int q = 0; q < cnt; ++q) {
              if (sid[q] == i) {
                acc += fmm_k64<KIND>(0.0, p0) * sbv[q];
                continue;
              }
              const float dx = (float)(sx[q] - xi[0]), dy = (float)(sy[q] - xi[1]),
                          dz = (float)(sz[q] - xi[2]);
              const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
              a = fmaf(fmm_k32<KIND>(d2, (float)p0), (float)sbv[q], a);
            }
            acc += (double)a;
          } else {
            for (int q = 0; q < cnt; ++q) {
              const double dx = sx[q] - xi[0], dy = sy[q] - xi[1], dz = sz[q] - xi[2];
              const double d2 = dx * dx + dy * dy + dz * dz;
              acc += fmm_k64<KIND>(d2, p0) * sbv[q];
            }
          }
        }
      }
    }
    if (act) c[i] = acc;
  }
}

// FP32 position of every particle relative to the centre of its leaf: the
// mixed-precision near field works on these small offsets (and on the
// leaf-to-leaf centre offsets), never on absolute FP32 coordinates.
__global__ void k_leaf_rel(int D, const int *__restrict__ leaves, const int *__restrict__ nb,
                           const int *__restrict__ ne, const double *__restrict__ box,
                           const double *__restrict__ pos, int64_t npos,
                           float4 *__restrict__ posf) {
  const int leaf = leaves[blockIdx.x];
  const double *bx = box + (size_t)leaf * 6;
  for (int i = nb[leaf] + threadIdx.x; i < ne[leaf]; i += blockDim.x) {
    float v[3] = {0.f, 0.f, 0.f};
    for (int d = 0; d < D; ++d)
      v[d] = (float)(pos[(int64_t)d * npos + i] - 0.5 * (bx[d] + bx[3 + d]));
    posf[i] = make_float4(v[0], v[1], v[2], 0.f);
  }
}

__device__ __forceinline__ float rsqrt_approx_f(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// FP32 kernel value of the mixed near field.  Laplace 1/(|dx| + p0) from the
// hardware reciprocal square root and reciprocal (~2 ulp each): |dx| =
// d2 * rsqrt(d2 + 1e-30), which is 0 at d2 = 0.
template <int KIND> __device__ __forceinline__ float p2p_k32(float d2, float p0) {
  if (KIND == ABX_K_LAPLACE) return rcp_approx_f(fmaf(d2, rsqrt_approx_f(d2 + 1e-30f), p0));
  return fmm_k32<KIND>(d2, p0);
}

constexpr int PT = 32;  // threads per target leaf (one warp) in the mixed near field
constexpr int PW = 4;   // target leaves (warps) per CTA

// Mixed-precision L2P + P2P: one warp per target leaf, one lane per target.
// L2P in FP32 from the leaf-relative FP32 position (x = offset /
// half-width): G of the leaf in FP32, the tensor-product sum nested by
// dimension (the node index is lexicographic, last dimension fastest), the
// innermost two levels in FP32 and the outermost in FP64; each source leaf of the near field is
// staged in shared memory as FP32 offsets from the target leaf's centre
// (leaf-relative FP32 position + FP32 centre offset), the pair terms are FP32
// with a staged chunk (<= 32 terms) summed in FP32 and chunks summed in
// FP64.  The self pair (a regularised singular kernel is huge there) is
// masked out of the FP32 sum and added in FP64.
template <int KIND>
__global__ void __launch_bounds__(PT * PW) k_l2p_p2p32(
    int D, int n, int ncheb, int nleaves, const int *__restrict__ leaves, const int *__restrict__ nb,
    const int *__restrict__ ne, const double *__restrict__ box, const float4 *__restrict__ posf,
    const float *__restrict__ b32, const double *__restrict__ b, const double *__restrict__ G,
    const int *__restrict__ rp, const int *__restrict__ src, double p0, const ChebTab32 tab,
    double *__restrict__ c) {
  __shared__ float sg_all[PW][MAXC];
  __shared__ float4 ss_all[PW][PT];
  __shared__ float sS_all[PW][3][MAXN][PT];  // per-lane Chebyshev values [d][m][lane]
  const int tid = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int li = blockIdx.x * PW + wl;
  if (li >= nleaves) return;  // whole warps: only warp-level synchronisation below
  float *sg = sg_all[wl];
  float4 *ss = ss_all[wl];
  const int leaf = leaves[li];
  const double *bx = box + (size_t)leaf * 6;
  double ct[3] = {0.0, 0.0, 0.0};
  float ihw[3] = {0.f, 0.f, 0.f};
  for (int d = 0; d < D; ++d) {
    ct[d] = 0.5 * (bx[d] + bx[3 + d]);
    const double hw = 0.5 * (bx[3 + d] - bx[d]);
    ihw[d] = hw > 0.0 ? (float)(1.0 / hw) : 0.f;
  }
  for (int j = tid; j < ncheb; j += PT) sg[j] = (float)G[(size_t)leaf * ncheb + j];
  __syncwarp();
  const float p0f = (float)p0;
  for (int i0 = nb[leaf]; i0 < ne[leaf]; i0 += PT) {
    const int i = i0 + tid;
    const bool act = i < ne[leaf];
    double acc = 0.0;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) {
      t = posf[i];
      const float xr[3] = {t.x, t.y, t.z};
      float S[MAXN];
      for (int d = 0; d < D; ++d) {
        cheb_sn_tab32(xr[d] * ihw[d], n, tab, S);
        for (int m = 0; m < n; ++m) sS_all[wl][d][m][tid] = S[m];
      }
      // sum_{m0} S0 sum_{m1} S1 sum_{m2} S2 g[m0, m1, m2] (D = 3; fewer levels below)
      const float(*sS)[MAXN][PT] = sS_all[wl];
      if (D == 3) {
        for (int m0 = 0; m0 < n; ++m0) {
          float p1 = 0.f;
          for (int m1 = 0; m1 < n; ++m1) {
            const float *gg = sg + (m0 * n + m1) * n;
            float p2 = 0.f;
            for (int m2 = 0; m2 < n; ++m2) p2 = fmaf(gg[m2], sS[2][m2][tid], p2);
            p1 = fmaf(p2, sS[1][m1][tid], p1);
          }
          acc += (double)(p1 * sS[0][m0][tid]);
        }
      } else if (D == 2) {
        for (int m0 = 0; m0 < n; ++m0) {
          float p1 = 0.f;
          for (int m1 = 0; m1 < n; ++m1) p1 = fmaf(sg[m0 * n + m1], sS[1][m1][tid], p1);
          acc += (double)(p1 * sS[0][m0][tid]);
        }
      } else {
        for (int m0 = 0; m0 < n; ++m0) acc += (double)(sg[m0] * sS[0][m0][tid]);
      }
    }
    for (int e = rp[li]; e < rp[li + 1]; ++e) {
      const int sl = src[e];
      const double *sbx = box + (size_t)sl * 6;
      float off[3] = {0.f, 0.f, 0.f};
      for (int d = 0; d < D; ++d) off[d] = (float)(0.5 * (sbx[d] + sbx[3 + d]) - ct[d]);
      const bool own = sl == leaf;
      for (int j0 = nb[sl]; j0 < ne[sl]; j0 += PT) {
        __syncwarp();
        const int j = j0 + tid;
        if (j < ne[sl]) {
          const float4 q = posf[j];
          ss[tid] = make_float4(q.x + off[0], q.y + off[1], q.z + off[2], b32[j]);
        }
        __syncwarp();
        const int cnt = min(PT, ne[sl] - j0);
        if (act) {
          float a = 0.f;
          if (own) {
            for (int q = 0; q < cnt; ++q) {
              const float4 sq = ss[q];
              const float dx = sq.x - t.x, dy = sq.y - t.y, dz = sq.z - t.z;
              const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
              const float w = j0 + q == i ? 0.f : p2p_k32<KIND>(d2, p0f);
              a = fmaf(w, sq.w, a);
            }
            if (i >= j0 && i < j0 + cnt) acc += fmm_k64<KIND>(0.0, p0) * b[i];
          } else {
#pragma unroll 4
            for (int q = 0; q < cnt; ++q) {
              const float4 sq = ss[q];
              const float dx = sq.x - t.x, dy = sq.y - t.y, dz = sq.z - t.z;
              const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
              a = fmaf(p2p_k32<KIND>(d2, p0f), sq.w, a);
            }
          }
          acc += (double)a;
        }
      }
    }
    if (act) c[i] = acc;
  }
}

// ------------------------------------------- FP64 near field on integers ---
__global__ void k_fixed_pos(int D, const double *__restrict__ pos, int64_t n, fx::Unit U,
                            longlong2 *__restrict__ fxy, long long *__restrict__ fz) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fxy[i] = make_longlong2(fx::to_fixed(pos[i], U.f, U.k),
                          D > 1 ? fx::to_fixed(pos[n + i], U.f, U.k) : 0);
  fz[i] = D > 2 ? fx::to_fixed(pos[2 * n + i], U.f, U.k) : 0;
}

// L2P in FP64: one warp per leaf, one lane per target, the tensor-product sum
// nested by dimension (n^3 + n^2 + n multiply-adds a target instead of 3 n^3
// products).
__global__ void __launch_bounds__(PT * PW) k_l2p64(
    int D, int n, int ncheb, int nleaves, const int *__restrict__ leaves, const int *__restrict__ nb,
    const int *__restrict__ ne, const double *__restrict__ box, const double *__restrict__ pos,
    int64_t npos, const double *__restrict__ G, const ChebTab tab, double *__restrict__ c) {
  __shared__ double sS_all[PW][3][MAXN][PT];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int li = blockIdx.x * PW + wl;
  if (li >= nleaves) return;  // whole warps: each lane reads its own column of sS only
  const int leaf = leaves[li];
  const double *bx = box + (size_t)leaf * 6;
  const double *g = G + (size_t)leaf * ncheb;
  double(*sS)[MAXN][PT] = sS_all[wl];
  for (int i = nb[leaf] + lane; i < ne[leaf]; i += PT) {
    for (int d = 0; d < D; ++d) {
      double S[MAXN];
      cheb_sn_tab(shift_coord(pos[(int64_t)d * npos + i], bx[d], bx[3 + d]), n, tab, S);
      for (int m = 0; m < n; ++m) sS[d][m][lane] = S[m];
    }
    double acc = 0.0;
    for (int m0 = 0; m0 < n; ++m0) {
      double p1 = 0.0;
      if (D == 1) {
        p1 = g[m0];
      } else {
        for (int m1 = 0; m1 < n; ++m1) {
          double p2 = 0.0;
          if (D == 2) {
            p2 = g[m0 * n + m1];
          } else {
            const double *gg = g + (m0 * n + m1) * n;
            for (int m2 = 0; m2 < n; ++m2) p2 = fma(gg[m2], sS[2][m2][lane], p2);
          }
          p1 = fma(p2, sS[1][m1][lane], p1);
        }
      }
      acc = fma(p1, sS[0][m0][lane], acc);
    }
    c[i] = acc;
  }
}

// Leaves an SM from which 4 warps work a leaf, below 16: 512 leaves (20,000 points
// in 3-D) 618 us the whole product with 4, 505 with 16; 1,024 (30,000 in 2-D) 303
// with 4, 374 with 16.
constexpr int64_t P2P_LEAVES4 = 5;
// P2P in FP64 accuracy on the integer units, added to the L2P result: WPL warps,
// a CTA, per target leaf, each taking every WPL-th tile of its sources; one lane
// per target.  Leaves hold 32 targets on average and
// a third of them a few more than 32: a last tile of r <= 16 targets is worked
// by 32 / p lanes a target (p the power of two above r), each taking every
// (32 / p)-th source, and the lanes' sums are added.  N = 1,048,576 uniform,
// Laplace, order 3: the whole product 57.2 -> 19.3 ms with this alone.
// With a warp a leaf few leaves left most of the GPU idle while a warp walked 400
// sources (12,934 points in 2-D, 581 -> 308 us the whole product), and many a
// last wave of long leaves (1,048,576 in 3-D, 10.9 -> 10.5 ms).
template <int KIND, int WPL>
__global__ void __launch_bounds__(PT * WPL) k_p2p_fix(
    int D, const int *__restrict__ leaves, const int *__restrict__ nb,
    const int *__restrict__ ne, const double *__restrict__ pos, int64_t npos,
    const longlong2 *__restrict__ fxy, const long long *__restrict__ fz,
    const double *__restrict__ b, const int *__restrict__ rp, const int *__restrict__ src, double p0,
    const fx::Consts C, double *__restrict__ c) {
  __shared__ longlong2 sxy_all[WPL][PT], szb_all[WPL][PT];
  __shared__ double part[WPL][PT];
  __shared__ fx::u64 tab[KIND == ABX_K_GAUSSIAN ? fx::EXP_TAB : 1];
  if (KIND == ABX_K_GAUSSIAN) {
    for (int i = threadIdx.x; i < fx::EXP_TAB; i += PT * WPL) tab[i] = fx::exp_table.v[i];
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int li = blockIdx.x;
  longlong2 *sxy = sxy_all[wl], *szb = szb_all[wl];
  const int leaf = leaves[li];
  for (int i0 = nb[leaf]; i0 < ne[leaf]; i0 += PT) {
    const int r = min(PT, ne[leaf] - i0);
    const int p = r > 16 ? 32 : r > 8 ? 16 : r > 4 ? 8 : 4;
    const int i = i0 + (lane & (p - 1)), grp = lane / p, ngrp = 32 / p;
    const bool act = (lane & (p - 1)) < r;
    long long x = 0, y = 0, z = 0;
    if (act) {
      const longlong2 f = fxy[i];
      x = fx::biased(f.x);
      y = fx::biased(f.y);
      z = fx::biased(fz[i]);
    }
    double acc = 0.0;
    int tile = 0;
    for (int e = rp[li]; e < rp[li + 1]; ++e) {
      const int sl = src[e];
      for (int j0 = nb[sl]; j0 < ne[sl]; j0 += PT) {
        if (tile++ % WPL != wl) continue;
        const int cnt = min(PT, ne[sl] - j0);
        __syncwarp();
        if (lane < cnt) {
          sxy[lane] = fxy[j0 + lane];
          szb[lane] = make_longlong2(fz[j0 + lane], __double_as_longlong(b[j0 + lane]));
        }
        __syncwarp();
        if (act) {
          for (int q = grp; q < cnt; q += ngrp) {
            const longlong2 s0 = sxy[q], s1 = szb[q];
            bool near;
            double v = fx::value<KIND>(fx::diff(s0.x, x), fx::diff(s0.y, y), fx::diff(s1.x, z), D, C,
                                       tab, near);
            if (KIND == ABX_K_LAPLACE && near) {
              int j = j0 + q;
              asm volatile("" : "+r"(j));  // (compared in here, not for every pair: 2 %)
              if (i != j) {
                double d2 = 0.0;
                for (int d = 0; d < D; ++d) {
                  const double dx = pos[(int64_t)d * npos + j] - pos[(int64_t)d * npos + i];
                  d2 += dx * dx;
                }
                v = fmm_k64<KIND>(d2, p0);
              }
            }
            acc = fma(v, __longlong_as_double(s1.y), acc);
          }
        }
      }
    }
    for (int o = p; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __syncthreads();
    part[wl][lane] = acc;
    __syncthreads();
    if (wl != 0) continue;
    for (int w = 1; w < WPL; ++w) acc += part[w][lane];
    if (act && grp == 0) c[i] += acc;
  }
}

// M2L matrices: for each (level box size, offset) K[i][j] = kernel(x_i^t, x_j^s)
template <int KIND>
__global__ void k_m2l_mats(int D, int n, int ncheb, const double *__restrict__ mat_desc,
                           const int *__restrict__ mi, double p0, double *__restrict__ Km) {
  // mat_desc per matrix: box size[3], offset[3] (source box lo - target box lo)
  const int m = blockIdx.y;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)ncheb * ncheb) return;
  const int i = (int)(e / ncheb), j = (int)(e % ncheb);
  const double *md = mat_desc + (size_t)m * 6;
  double d2 = 0.0;
  for (int d = 0; d < D; ++d) {
    const double h = md[d];
    const double pi = 0.5 * (cheb_node(mi[i * 3 + d], n) + 1) * h;
    const double pj = 0.5 * (cheb_node(mi[j * 3 + d], n) + 1) * h + md[3 + d];
    const double dx = pj - pi;
    d2 += dx * dx;
  }
  Km[(size_t)m * ncheb * ncheb + e] = fmm_k64<KIND>(d2, p0);
}

}  // namespace

// ----------------------------------------------------------- plan build ---
// eta scales the admissibility of a box pair: it is near (P2P or further
// refinement) iff (max diameter)^2 > eta^2 (box distance)^2; eta = 1 is the
// reference FMM's theta_condition (src/detail/FastMultipoleMethod.h:1249-1279).
int fmm_plan_build(abx_operator *op, int order, FmmPlan *&out, double eta = 1.0) {
  abx_particles *p = op->rows;
  abx_context *ctx = p->ctx;
  cudaStream_t s = ctx->stream;
  ABX_REQUIRE(p->searchable && p->search_kind == 1, ABX_ERR_STATE,
              "the FMM needs an octree: call abx_particles_init_octree first");
  ABX_REQUIRE(order >= 2 && order <= MAXN, ABX_ERR_INVALID, "Chebyshev order must be in 2..%d", MAXN);
  const auto t0 = std::chrono::steady_clock::now();
  const OctTree &T = p->tree;
  FmmPlan *P = new FmmPlan();
  const int D = p->dim;
  P->D = D;
  P->n = order;
  P->tab = cheb_table(order);
  P->tab32 = cheb_table32(P->tab);
  P->nchild = 1 << D;
  P->ncheb = 1;
  for (int d = 0; d < D; ++d) P->ncheb *= order;
  P->kind = op->k.kind;
  P->p0 = op->k.p[0];
  const int nc = P->ncheb;
  P->mi.assign((size_t)nc * 3, 0);
  for (int j = 0; j < nc; ++j) {
    int r = j;
    for (int d = D - 1; d >= 0; --d) {
      P->mi[j * 3 + d] = r % order;
      r /= order;
    }
  }
  const int NN = (int)T.tag.size();
  P->nnodes = NN;
  std::vector<double> boxes((size_t)NN * 6, 0.0);
  for (int nd = 0; nd < NN; ++nd) {
    double lo[3] = {0, 0, 0}, hi[3] = {1, 1, 1};
    T.box(p->grid, nd, lo, hi);
    for (int d = 0; d < 3; ++d) {
      boxes[nd * 6 + d] = d < D ? lo[d] : 0.0;
      boxes[nd * 6 + 3 + d] = d < D ? hi[d] : 1.0;
    }
  }
  // ---- traversal on the device: M2L pairs grouped by matrix key, P2P lists
  DevBuf<double> boxes_d;
  if (int e = boxes_d.reserve(boxes.size() + 1)) {
    delete P;
    return e;
  }
  if (!boxes.empty())
    cudaMemcpyAsync(boxes_d.ptr, boxes.data(), boxes.size() * 8, cudaMemcpyHostToDevice, s);
  FmmLists lists;
  if (NN > 1) {
    const int e = fmm_traverse_device(p, boxes_d.ptr, eta, lists);
    if (e != ABX_OK) {
      delete P;
      return e;
    }
  } else {
    lists.mat_off.assign(1, 0);
  }
  // ---- links by level, octant-major (M2M bottom-up uses deepest first)
  std::vector<std::array<int, 3>> links;  // parent, child, octant
  int maxlev = 0;
  {
    const OctDev &O = p->oct;
    for (size_t L = 1; L < O.lvl_base.size(); ++L)
      for (int c = 0; c < O.lvl_count[L]; ++c) {
        const int t = O.lvl_base[L] + c;
        if (T.kind[t] == 0) continue;
        links.push_back({T.parent[t], t, c % P->nchild});
        maxlev = std::max(maxlev, (int)L);
      }
  }
  std::vector<int> flat;
  std::vector<int2> batches;
  P->batch_off.assign(maxlev + 2, 0);
  P->batch_cnt.assign(maxlev + 2, 0);
  {
    std::vector<std::vector<std::vector<int>>> by(maxlev + 1,
                                                  std::vector<std::vector<int>>(P->nchild));
    for (size_t q = 0; q < links.size(); ++q)
      by[T.level[links[q][1]]][links[q][2]].push_back((int)q);
    for (int lev = 1; lev <= maxlev; ++lev) {
      P->batch_off[lev] = (int)batches.size();
      // octant-major within the level: batches of <= NBL links share a matrix
      for (int o = 0; o < P->nchild; ++o) {
        int run = 0;
        for (int q : by[lev][o]) {
          const int idx = (int)(flat.size() / 3);
          if (run == 0) batches.push_back(make_int2(idx, 0));
          ++batches.back().y;
          run = (run + 1) % NBL;
          flat.push_back(links[q][0]);
          flat.push_back(links[q][1]);
          flat.push_back(links[q][2]);
        }
      }
      P->batch_cnt[lev] = (int)batches.size() - P->batch_off[lev];
    }
  }
  // ---- M2L matrices: (level, offset) keys from the traversal, the box size
  // of a representative target
  std::vector<double> mdesc;
  P->nmat = (int)lists.mat_key.size();
  P->n_m2l = (int)lists.n_m2l;
  for (int m = 0; m < P->nmat; ++m) {
    const int t = lists.mat_rep[m];
    double hbox[3] = {1, 1, 1};
    for (int d = 0; d < D; ++d) hbox[d] = boxes[t * 6 + 3 + d] - boxes[t * 6 + d];
    for (int d = 0; d < 3; ++d) mdesc.push_back(hbox[d]);
    for (int d = 0; d < 3; ++d)
      mdesc.push_back(d < D ? (double)lists.mat_key[m][1 + d] * hbox[d] : 0.0);
  }
  P->mat_off = lists.mat_off;
  std::vector<int> leaves = T.leaves;
  P->nleaves = (int)leaves.size();
  // near field in fixed point: two near boxes of one level are no larger than
  // the largest leaf (of sides s_d) and less than max(s) / eta apart, so their
  // points differ by less than 2 s_d + max(s) / eta in every dimension
  {
    double side[3] = {0, 0, 0}, reach2 = 0.0;
    for (int leaf : leaves)
      for (int d = 0; d < D; ++d)
        side[d] = std::max(side[d], boxes[leaf * 6 + 3 + d] - boxes[leaf * 6 + d]);
    const double gap = std::max(side[0], std::max(side[1], side[2])) / std::min(eta, 1.0);
    for (int d = 0; d < D; ++d) {
      const double most = std::min(2.0 * side[d] + gap, p->grid.hi[d] - p->grid.lo[d]);
      reach2 += most * most;
    }
    const double reach = std::sqrt(reach2) * (1.0 + 1e-6);
    switch (P->kind) {
    case ABX_K_LAPLACE: P->unit = fx::make_unit<fx::LAPLACE>(P->p0, reach); break;
    case ABX_K_GAUSSIAN:
    case ABX_K_COMPACT_GAUSSIAN: P->unit = fx::make_unit<fx::GAUSSIAN>(P->p0, reach); break;
    case ABX_K_MULTIQUADRIC: P->unit = fx::make_unit<fx::MULTIQUADRIC>(P->p0, reach); break;
    default: break;
    }
  }
  // ---- child interpolation matrices Tc[o][i][j] = R_i(node j of child o; parent box)
  std::vector<double> Tc((size_t)P->nchild * nc * nc);
  for (int o = 0; o < P->nchild; ++o)
    for (int j = 0; j < nc; ++j) {
      double S[3][MAXN];
      for (int d = 0; d < D; ++d) {
        const int bit = (o >> (D - 1 - d)) & 1;  // child box in the unit parent box [-1,1]
        const double clo = bit ? 0.0 : -1.0, chi = bit ? 1.0 : 0.0;
        const double x = 0.5 * (cheb_node(P->mi[j * 3 + d], order) + 1) * (chi - clo) + clo;
        cheb_sn(x, order, S[d]);
      }
      for (int i = 0; i < nc; ++i) {
        double r = 1.0;
        for (int d = 0; d < D; ++d) r *= S[d][P->mi[i * 3 + d]];
        Tc[((size_t)o * nc + i) * nc + j] = r;
      }
    }
  // ---- device upload
  int st;
  auto fail = [&](int e) {
    delete P;
    return e;
  };
  std::vector<int> nb(NN), ne(NN);
  for (int nd = 0; nd < NN; ++nd) {
    nb[nd] = T.begin[nd];
    ne[nd] = T.end[nd];
  }
  if ((st = P->W.reserve((size_t)NN * nc)) || (st = P->G.reserve((size_t)NN * nc)) ||
      (st = P->Tc.reserve(Tc.size())) || (st = P->box.reserve(boxes.size())) ||
      (st = P->leaf_ids.reserve(leaves.size() + 1)) || (st = P->node_begin.reserve(NN)) ||
      (st = P->node_end.reserve(NN)) || (st = P->links.reserve(flat.size() + 1)) ||
      (st = P->batches.reserve(batches.size() + 1)) || (st = P->TcT.reserve(Tc.size())) ||
      (st = P->Km.reserve((size_t)std::max(1, P->nmat) * nc * nc)) ||
      (st = P->mat_off_d.reserve(P->nmat + 1)))
    return fail(st);
  // the traversal's device lists move into the plan
  auto take = [](auto &dst, auto &src) {
    std::swap(dst.ptr, src.ptr);
    std::swap(dst.cap, src.cap);
  };
  take(P->m2l_by_mat, lists.m2l_by_mat);
  take(P->p2p_rowptr, lists.p2p_rowptr);
  take(P->p2p_src, lists.p2p_src);
  if ((st = P->m2l_by_mat.reserve(1)) ||
      (st = P->p2p_rowptr.reserve(1)) || (st = P->p2p_src.reserve(1)))
    return fail(st);
  if (NN <= 1) {
    const int zero = 0;
    cudaMemcpyAsync(P->p2p_rowptr.ptr, &zero, 4, cudaMemcpyHostToDevice, s);
  }
  DevBuf<double> md_d;
  if ((st = P->mi_d.reserve(P->mi.size())) || (st = md_d.reserve(mdesc.size() + 1))) return fail(st);
  // tensor-core M2L tiles: 64 pairs for the mma.sync kernel (<= 64 nodes),
  // t5_pairs pairs for the tcgen05 kernel, of one matrix each
  std::vector<int> tmat, tfirst;
  const int tile_pairs = P->tile_pairs = nc <= 64 ? TC_PAIRS : t5_pairs((nc + 127) / 128);
  for (int m = 0; m < P->nmat; ++m)
    for (int q = P->mat_off[m]; q < P->mat_off[m + 1]; q += tile_pairs) {
      tmat.push_back(m);
      tfirst.push_back(q);
    }
  P->ntiles = (int)tmat.size();
  if ((st = P->tile_mat.reserve(tmat.size() + 1)) || (st = P->tile_first.reserve(tfirst.size() + 1)))
    return fail(st);
  auto up = [&](void *dst, const void *src, size_t bytes) {
    if (bytes) cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  };
  up(P->Tc.ptr, Tc.data(), Tc.size() * 8);
  if (!Tc.empty())
    k_transpose_tc<double><<<ceil_div(Tc.size(), 256), 256, 0, s>>>(P->Tc.ptr, P->nchild, nc,
                                                                   P->TcT.ptr);
  up(P->box.ptr, boxes.data(), boxes.size() * 8);
  up(P->leaf_ids.ptr, leaves.data(), leaves.size() * 4);
  up(P->node_begin.ptr, nb.data(), nb.size() * 4);
  up(P->node_end.ptr, ne.data(), ne.size() * 4);
  up(P->links.ptr, flat.data(), flat.size() * 4);
  up(P->batches.ptr, batches.data(), batches.size() * sizeof(int2));
  up(P->mat_off_d.ptr, P->mat_off.data(), P->mat_off.size() * 4);
  up(P->mi_d.ptr, P->mi.data(), P->mi.size() * 4);
  up(P->tile_mat.ptr, tmat.data(), tmat.size() * 4);
  up(P->tile_first.ptr, tfirst.data(), tfirst.size() * 4);
  up(md_d.ptr, mdesc.data(), mdesc.size() * 8);
  if (P->nmat > 0) {
    dim3 grid(ceil_div((size_t)nc * nc, 256), P->nmat);
    switch (P->kind) {
    case ABX_K_LAPLACE: k_m2l_mats<ABX_K_LAPLACE><<<grid, 256, 0, s>>>(D, order, nc, md_d.ptr, P->mi_d.ptr, P->p0, P->Km.ptr); break;
    case ABX_K_GAUSSIAN: k_m2l_mats<ABX_K_GAUSSIAN><<<grid, 256, 0, s>>>(D, order, nc, md_d.ptr, P->mi_d.ptr, P->p0, P->Km.ptr); break;
    case ABX_K_COMPACT_GAUSSIAN: k_m2l_mats<ABX_K_COMPACT_GAUSSIAN><<<grid, 256, 0, s>>>(D, order, nc, md_d.ptr, P->mi_d.ptr, P->p0, P->Km.ptr); break;
    case ABX_K_MULTIQUADRIC: k_m2l_mats<ABX_K_MULTIQUADRIC><<<grid, 256, 0, s>>>(D, order, nc, md_d.ptr, P->mi_d.ptr, P->p0, P->Km.ptr); break;
    case ABX_K_CONST: k_m2l_mats<ABX_K_CONST><<<grid, 256, 0, s>>>(D, order, nc, md_d.ptr, P->mi_d.ptr, P->p0, P->Km.ptr); break;
    default:
      set_error("FMM: kernel kind %d not supported", P->kind);
      return fail(ABX_ERR_INVALID);
    }
  }
  if (P->nleaves > 0) {
    if ((st = P->posf.reserve((size_t)std::max<int64_t>(op->rows->n, 1)))) return fail(st);
    k_leaf_rel<<<P->nleaves, FT, 0, s>>>(D, P->leaf_ids.ptr, P->node_begin.ptr, P->node_end.ptr,
                                          P->box.ptr, op->rows->pos.ptr, op->rows->n, P->posf.ptr);
  }
  if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    set_error("FMM plan upload failed");
    return fail(ABX_ERR_CUDA);
  }
  P->max_level.assign(1, maxlev);
  P->sms = std::max(ctx->num_sms, 1);
  P->build_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  out = P;
  return ABX_OK;
}

namespace {
// The integer near field's positions.
int p2p_fix_prepare(FmmPlan *P, int64_t npos) {
  ABX_TRY(P->fz.reserve((size_t)npos));
  return P->fxy.reserve((size_t)npos);
}

template <int KIND>
int launch_l2p_p2p(FmmPlan *P, cudaStream_t s, const double *pos, int64_t npos, const double *b,
                   double *c, bool mixed) {
  if (mixed) {
    // P->b32 holds this matvec's FP32 weights (converted before the P2M)
    k_l2p_p2p32<KIND><<<ceil_div((size_t)P->nleaves, PW), PT * PW, 0, s>>>(
        P->D, P->n, P->ncheb, P->nleaves, P->leaf_ids.ptr, P->node_begin.ptr, P->node_end.ptr,
        P->box.ptr, P->posf.ptr, P->b32.ptr, b, P->G.ptr, P->p2p_rowptr.ptr, P->p2p_src.ptr,
        P->p0, P->tab32, c);
  } else if (KIND != ABX_K_CONST && P->unit.ok &&
             (P->fxy.cap >= (size_t)npos || !stream_capturing(s))) {
    constexpr int FK = KIND == ABX_K_COMPACT_GAUSSIAN || KIND == ABX_K_CONST ? ABX_K_GAUSSIAN : KIND;
    ABX_TRY(p2p_fix_prepare(P, npos));
    const unsigned lb = ceil_div((size_t)P->nleaves, PW);
    k_fixed_pos<<<ceil_div((size_t)npos, 256), 256, 0, s>>>(P->D, pos, npos, P->unit, P->fxy.ptr,
                                                            P->fz.ptr);
    k_l2p64<<<lb, PT * PW, 0, s>>>(P->D, P->n, P->ncheb, P->nleaves, P->leaf_ids.ptr,
                                   P->node_begin.ptr, P->node_end.ptr, P->box.ptr, pos, npos,
                                   P->G.ptr, P->tab, c);
    auto p2p = [&](auto kernel, int threads) {
      kernel<<<P->nleaves, threads, 0, s>>>(P->D, P->leaf_ids.ptr, P->node_begin.ptr,
                                        P->node_end.ptr, pos, npos, P->fxy.ptr, P->fz.ptr, b,
                                        P->p2p_rowptr.ptr, P->p2p_src.ptr, P->p0,
                                        fx::consts(P->unit, 1.0 / P->p0), c);
    };
    if (P->nleaves >= P->sms * P2P_LEAVES4)
      p2p(k_p2p_fix<FK, 4>, PT * 4);
    else
      p2p(k_p2p_fix<FK, 16>, PT * 16);
  } else
    k_l2p_p2p<KIND, false><<<P->nleaves, FT, 0, s>>>(
        P->D, P->n, P->ncheb, P->leaf_ids.ptr, P->node_begin.ptr, P->node_end.ptr, P->box.ptr, pos,
        npos, b, P->mi_d.ptr, P->G.ptr, P->p2p_rowptr.ptr, P->p2p_src.ptr, P->p0, P->tab, c);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}
}  // namespace

// One level's M2M or L2L.  Threads a row (k_m2m_l2l): four below the line, one from it
// on.  Measured in us, M2M / L2L, four against one, 152 SMs:
//   FP32    64 CTAs   21 / 18 against 26 / 23       FP64    64   40 / 37 against 63 / 59
//          240        44 / 40 against 58 / 54               192  161 / 158 against 174 / 169
//          512        33 / 17 against 25 / 22             1,024  355 / 351 against 392 / 374
//        1,024        75 / 49 against 38 / 34             1,536  855 / 849 against 875 / 869
//        1,536       148 / 110 against 62 / 58            4,096  886 / 875 against 861 / 849
// (orders 5 to 7; FP64's line is at 8 CTAs an SM because with few nodes one thread is the
// faster before: 2-D, order 3, 2,048 CTAs, a product 1,398 us against 1,437).
template <typename T, bool M2M>
void launch_links(const FmmPlan *P, int lev, const T *mats, double *V, cudaStream_t s) {
  if (P->batch_cnt[lev] == 0) return;
  const dim3 grid(P->batch_cnt[lev], ceil_div(P->ncheb, FT));
  const int2 *bt = P->batches.ptr + P->batch_off[lev];
  constexpr int64_t LINE = sizeof(T) == 4 ? 2 : 8;  // CTAs an SM
  if ((int64_t)grid.x * grid.y < LINE * P->sms)
    k_m2m_l2l<T, M2M, 4><<<grid, 4 * FT, 0, s>>>(P->ncheb, P->links.ptr, bt, mats, V);
  else
    k_m2m_l2l<T, M2M, 1><<<grid, FT, 0, s>>>(P->ncheb, P->links.ptr, bt, mats, V);
}

namespace {
// The FP64 M2L's tiles, split matrices and buffers, once per plan.
int m2l64_prepare(FmmPlan *P, cudaStream_t s) {
  const int nc = P->ncheb, chunks = (nc + MF_K - 1) / MF_K;
  if (P->m2l64_ready) return ABX_OK;
  DevBuf<int> span_d;
  std::vector<int> span((size_t)P->nmat);
  ABX_TRY(span_d.reserve(span.size()));
  k_row_span<<<P->nmat, MF_T, 0, s>>>(P->Km.ptr, nc, span_d.ptr);
  ABX_CHECK_CUDA(cudaGetLastError());
  ABX_CHECK_CUDA(cudaMemcpyAsync(span.data(), span_d.ptr, span.size() * 4, cudaMemcpyDeviceToHost, s));
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));
  std::vector<int> mat[2], first[2];  // by digits, in FP64
  for (int m = 0; m < P->nmat; ++m) {
    const int wide = span[m] > fx::ONE_SIZE, tile = wide ? MW_PAIRS : mf_pairs(nc);
    for (int q = P->mat_off[m]; q < P->mat_off[m + 1]; q += tile) {
      mat[wide].push_back(m);
      first[wide].push_back(q);
    }
  }
  auto up = [&](DevBuf<int> &dst, const std::vector<int> &v) -> int {
    ABX_TRY(dst.reserve(v.size() + 1));
    ABX_CHECK_CUDA(cudaMemcpyAsync(dst.ptr, v.data(), v.size() * 4, cudaMemcpyHostToDevice, s));
    return ABX_OK;
  };
  ABX_TRY(up(P->mf_mat, mat[0]));
  ABX_TRY(up(P->mf_first, first[0]));
  ABX_TRY(up(P->mw_mat, mat[1]));
  ABX_TRY(up(P->mw_first, first[1]));
  P->mf_tiles = (int)mat[0].size();
  P->mw_tiles = (int)mat[1].size();
  if (P->mf_tiles > 0) {
    const int64_t rows = (int64_t)P->nmat * nc;
    ABX_TRY(P->ke.reserve((size_t)rows));
    ABX_TRY(P->Kd.reserve((size_t)rows * chunks * MF_ROW));
    k_split_digits<<<ceil_div((size_t)rows, 8), 256, 0, s>>>(P->Km.ptr, rows, nc, nc, P->Kd.ptr,
                                                             P->ke.ptr);
    ABX_CHECK_CUDA(cudaGetLastError());
    ABX_TRY(P->Wd.reserve((size_t)P->nnodes * chunks * MF_ROW));
    ABX_TRY(P->we.reserve((size_t)P->nnodes));
  }
  ABX_CHECK_CUDA(cudaStreamSynchronize(s));  // the host lists end here
  P->m2l64_ready = true;
  return ABX_OK;
}

// G += K W in FP64.
int m2l64(FmmPlan *P, cudaStream_t s) {
  const int nc = P->ncheb;
  auto by_fp64 = [&](const int *mat, const int *first, int tiles, int pairs) {
    k_m2l64<<<tiles, FT, 0, s>>>(nc, P->Km.ptr, P->m2l_by_mat.ptr, P->mat_off_d.ptr, mat, first,
                                 pairs, P->W.ptr, P->G.ptr);
  };
  if (!P->m2l64_ready && stream_capturing(s)) {
    by_fp64(P->tile_mat.ptr, P->tile_first.ptr, P->ntiles, P->tile_pairs);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  ABX_TRY(m2l64_prepare(P, s));
  if (P->mw_tiles > 0) by_fp64(P->mw_mat.ptr, P->mw_first.ptr, P->mw_tiles, MW_PAIRS);
  ABX_CHECK_CUDA(cudaGetLastError());
  if (P->mf_tiles == 0) return ABX_OK;
  k_split_digits<<<ceil_div((size_t)P->nnodes, 8), 256, 0, s>>>(P->W.ptr, P->nnodes, nc, 1, P->Wd.ptr,
                                                                P->we.ptr);
  auto run = [&](auto kern, int tr, size_t smem) -> int {
    ABX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<dim3(P->mf_tiles, (nc + tr - 1) / tr), MF_T, smem, s>>>(
        nc, P->Kd.ptr, P->ke.ptr, P->Wd.ptr, P->we.ptr, P->m2l_by_mat.ptr, P->mat_off_d.ptr,
        P->mf_mat.ptr, P->mf_first.ptr, P->G.ptr);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  };
  // up to 32 nodes: one stage, 32 rows
  return nc <= 32 ? run(k_m2l_fix<32, 64, 1>, 32, mf_stage<32, 64>())
                  : run(k_m2l_fix<64, 32, 2>, 64, 2 * mf_stage<64, 32>());
}
}  // namespace

// What a plan's FP64 products keep: a first product then allocates nothing and
// waits for nothing.  (Without it, one that is captured runs the FP64 kernels.)
int fmm_plan_prepare(FmmPlan *P, int64_t npos, cudaStream_t s) {
  if (P->unit.ok) ABX_TRY(p2p_fix_prepare(P, npos));
  return P->n_m2l > 0 ? m2l64_prepare(P, s) : ABX_OK;
}

// c = K b through the five FMM passes (storage order of the octree set).
int fmm_matvec_device(abx_operator *op, const double *b, double *c) {
  FmmPlan *P = op->fmm;
  abx_particles *p = op->rows;
  cudaStream_t s = p->ctx->stream;
  const int nc = P->ncheb;
  const int64_t npos = p->n;
  if (npos == 0) return ABX_OK;
  const bool mixed = op->precision == ABX_PREC_MIXED;
  ABX_CHECK_CUDA(cudaMemsetAsync(P->W.ptr, 0, (size_t)P->nnodes * nc * 8, s));
  ABX_CHECK_CUDA(cudaMemsetAsync(P->G.ptr, 0, (size_t)P->nnodes * nc * 8, s));
  if (mixed) {
    ABX_TRY(P->b32.reserve((size_t)npos));
    k_f64_to_f32<<<ceil_div((size_t)npos, 256), 256, 0, s>>>(b, npos, P->b32.ptr);
    if (!P->Tc32.ptr) {
      const size_t nt = (size_t)P->nchild * nc * nc;
      ABX_TRY(P->Tc32.reserve(nt));
      ABX_TRY(P->Tc32T.reserve(nt));
      k_f64_to_f32<<<ceil_div(nt, 256), 256, 0, s>>>(P->Tc.ptr, nt, P->Tc32.ptr);
      k_transpose_tc<float><<<ceil_div(nt, 256), 256, 0, s>>>(P->Tc.ptr, P->nchild, nc,
                                                             P->Tc32T.ptr);
    }
  }
  if (P->nleaves > 0) {
    if (mixed)
      k_p2m32<<<P->nleaves, FT, 0, s>>>(P->D, P->n, nc, P->leaf_ids.ptr, P->node_begin.ptr,
                                        P->node_end.ptr, P->box.ptr, P->posf.ptr, P->b32.ptr,
                                        P->mi_d.ptr, P->tab32, P->W.ptr);
    else
      k_p2m<<<P->nleaves, FT, 0, s>>>(P->D, P->n, nc, P->leaf_ids.ptr, P->node_begin.ptr,
                                      P->node_end.ptr, P->box.ptr, p->pos.ptr, npos, b,
                                      P->mi_d.ptr, P->tab, P->W.ptr);
  }
  const int maxlev = P->max_level.empty() ? 0 : P->max_level[0];
  for (int lev = maxlev; lev >= 1; --lev) {
    if (mixed) launch_links<float, true>(P, lev, P->Tc32T.ptr, P->W.ptr, s);
    else launch_links<double, true>(P, lev, P->TcT.ptr, P->W.ptr, s);
  }
  ABX_CHECK_CUDA(cudaGetLastError());
  if (P->n_m2l > 0) {
    if (mixed) {
      const size_t tot = (size_t)P->nnodes * nc;
      const int ldg = (nc + 3) / 4 * 4;
      const int ldk = (nc + 31) / 32 * 32;
      ABX_TRY(P->G32.reserve((size_t)P->nnodes * ldg));
      ABX_CHECK_CUDA(cudaMemsetAsync(P->G32.ptr, 0, (size_t)P->nnodes * ldg * 4, s));
      if (nc <= 64) {
        // mma.sync tiles (a 128-row tcgen05 tile would be mostly padding)
        if (!P->Kmh.ptr) {
          const size_t nk = (size_t)P->nmat * nc * ldk;
          ABX_TRY(P->Kmh.reserve(nk));
          ABX_TRY(P->Kml.reserve(nk));
          k_split_tf32<<<ceil_div(nk, 256), 256, 0, s>>>(P->Km.ptr, (int64_t)P->nmat * nc, nc,
                                                         ldk, P->Kmh.ptr, P->Kml.ptr);
        }
        ABX_TRY(P->W32.reserve((size_t)P->nnodes * ldk));
        k_to_f32_padded<<<ceil_div((size_t)P->nnodes * ldk, 256), 256, 0, s>>>(
            P->W.ptr, P->nnodes, nc, ldk, P->W32.ptr);
        auto launch_m2l = [&](auto kern, int mt, int threads, size_t smem) -> int {
          ABX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
          const dim3 grid(P->ntiles, (nc + mt - 1) / mt);
          kern<<<grid, threads, smem, s>>>(nc, ldk, ldg, P->Kmh.ptr, P->Kml.ptr,
                                           P->m2l_by_mat.ptr, P->mat_off_d.ptr, P->tile_mat.ptr,
                                           P->tile_first.ptr, P->W32.ptr, P->G32.ptr);
          return ABX_OK;
        };
        if (nc <= 32)
          ABX_TRY(launch_m2l(k_m2l_tc2<1>, M2Cfg<1>::MT, M2Cfg<1>::THREADS, M2Cfg<1>::SMEM));
        else
          ABX_TRY(launch_m2l(k_m2l_tc2<2>, M2Cfg<2>::MT, M2Cfg<2>::THREADS, M2Cfg<2>::SMEM));
      } else {
        // 5th-generation tensor cores (tcgen05, TMEM accumulators)
        const int nkb = (nc + T5_KB - 1) / T5_KB;
        const int nrb = (nc + 127) / 128;  // 1..4 for orders 5..8
        if (!P->Kp.ptr) {
          const size_t nk = (size_t)P->nmat * nkb * nrb * 2 * (T5_PART / 2);
          ABX_TRY(P->Kp.reserve(nk));
          ABX_TRY(P->Kp_scale.reserve(P->nmat));
          k_mat_scale<<<P->nmat, KS_TPB, 0, s>>>(P->Km.ptr, (int64_t)nc * nc, P->Kp_scale.ptr);
          k_pack_f16<<<ceil_div(nk, 256), 256, 0, s>>>(P->Km.ptr, P->Kp_scale.ptr, P->nmat, nc, nkb,
                                                       nrb, P->Kp.ptr);
        }
        ABX_TRY(P->W16h.reserve((size_t)P->nnodes * ldk));
        ABX_TRY(P->W16l.reserve((size_t)P->nnodes * ldk));
        ABX_TRY(P->W16_scale.reserve(P->nnodes));
        k_split_f16<<<ceil_div(P->nnodes, 8), 256, 0, s>>>(P->W.ptr, P->nnodes, nc, ldk, P->W16h.ptr,
                                                           P->W16l.ptr, P->W16_scale.ptr);
        int *status = p->ctx->dev_flag.ptr + 8;
        ABX_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int), s));
        auto launch_tc5 = [&](auto kern, size_t smem) -> int {
          ABX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
          kern<<<P->ntiles, 128, smem, s>>>(nc, nkb, ldk, ldg, P->Kp.ptr, P->Kp_scale.ptr, P->m2l_by_mat.ptr,
                                            P->mat_off_d.ptr, P->tile_mat.ptr, P->tile_first.ptr,
                                            P->W16h.ptr, P->W16l.ptr, P->W16_scale.ptr, P->G32.ptr, status,
                                            (uint64_t)(P->wait_limit_s * 1e9), P->drop_arrive);
          return ABX_OK;
        };
        switch (nrb) {
          case 1: ABX_TRY(launch_tc5(k_m2l_tc5<1>, T5Cfg<1>::SMEM)); break;
          case 2: ABX_TRY(launch_tc5(k_m2l_tc5<2>, T5Cfg<2>::SMEM)); break;
          case 3: ABX_TRY(launch_tc5(k_m2l_tc5<3>, T5Cfg<3>::SMEM)); break;
          default: ABX_TRY(launch_tc5(k_m2l_tc5<4>, T5Cfg<4>::SMEM)); break;
        }
        ABX_CHECK_CUDA(cudaGetLastError());
        int st = 0;
        ABX_CHECK_CUDA(cudaMemcpyAsync(&st, status, sizeof(int), cudaMemcpyDeviceToHost, s));
        ABX_CHECK_CUDA(cudaStreamSynchronize(s));
        ABX_REQUIRE(st == 0, ABX_ERR_TIMEOUT, "FMM M2L: a tensor-core completion wait timed out");
      }
      k_add_g32<<<ceil_div(tot, 256), 256, 0, s>>>(P->G32.ptr, P->nnodes, nc, ldg, P->G.ptr);
    } else {
      ABX_TRY(m2l64(P, s));
    }
    ABX_CHECK_CUDA(cudaGetLastError());
  }
  for (int lev = 1; lev <= maxlev; ++lev) {
    if (mixed) launch_links<float, false>(P, lev, P->Tc32.ptr, P->G.ptr, s);
    else launch_links<double, false>(P, lev, P->Tc.ptr, P->G.ptr, s);
  }
  ABX_CHECK_CUDA(cudaGetLastError());
  if (P->nleaves == 0) return ABX_OK;
  switch (P->kind) {
  case ABX_K_LAPLACE: return launch_l2p_p2p<ABX_K_LAPLACE>(P, s, p->pos.ptr, npos, b, c, mixed);
  case ABX_K_GAUSSIAN: return launch_l2p_p2p<ABX_K_GAUSSIAN>(P, s, p->pos.ptr, npos, b, c, mixed);
  case ABX_K_COMPACT_GAUSSIAN:
    return launch_l2p_p2p<ABX_K_COMPACT_GAUSSIAN>(P, s, p->pos.ptr, npos, b, c, mixed);
  case ABX_K_MULTIQUADRIC:
    return launch_l2p_p2p<ABX_K_MULTIQUADRIC>(P, s, p->pos.ptr, npos, b, c, mixed);
  case ABX_K_CONST: return launch_l2p_p2p<ABX_K_CONST>(P, s, p->pos.ptr, npos, b, c, mixed);
  }
  set_error("FMM: unsupported kernel");
  return ABX_ERR_INVALID;
}

}  // namespace abx

using namespace abx;

extern "C" int abx_create_fmm_operator(abx_particles *p, const abx_kernel *k, int order,
                                       abx_operator **out) {
  ABX_REQUIRE(p && k && out, ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(k->kind == ABX_K_LAPLACE || k->kind == ABX_K_GAUSSIAN ||
                  k->kind == ABX_K_COMPACT_GAUSSIAN || k->kind == ABX_K_MULTIQUADRIC ||
                  k->kind == ABX_K_CONST,
              ABX_ERR_INVALID, "FMM: kernel kind %d not supported", k->kind);
  ABX_TRY(ctx_activate(p->ctx));
  abx_operator *op = new abx_operator();
  op->kind = 2;
  op->rows = p;
  op->cols = p;
  op->k = *k;
  FmmPlan *P = nullptr;
  const int st = fmm_plan_build(op, order, P);
  if (st != ABX_OK) {
    delete op;
    return st;
  }
  op->fmm = P;
  particles_retain(p);
  particles_retain(p);
  *out = op;
  return ABX_OK;
}

extern "C" int abx_create_h2_operator(abx_particles *p, const abx_kernel *k, int order,
                                      double eta, abx_operator **out) {
  ABX_REQUIRE(p && k && out, ABX_ERR_INVALID, "null argument");
  ABX_REQUIRE(eta > 0.0 && std::isfinite(eta), ABX_ERR_INVALID, "eta must be positive");
  ABX_REQUIRE(k->kind == ABX_K_LAPLACE || k->kind == ABX_K_GAUSSIAN ||
                  k->kind == ABX_K_COMPACT_GAUSSIAN || k->kind == ABX_K_MULTIQUADRIC ||
                  k->kind == ABX_K_CONST,
              ABX_ERR_INVALID, "H2: kernel kind %d not supported", k->kind);
  ABX_TRY(ctx_activate(p->ctx));
  abx_operator *op = new abx_operator();
  op->kind = 2;
  op->rows = p;
  op->cols = p;
  op->k = *k;
  FmmPlan *P = nullptr;
  const int st = fmm_plan_build(op, order, P, eta);
  if (st != ABX_OK) {
    delete op;
    return st;
  }
  op->fmm = P;
  particles_retain(p);
  particles_retain(p);
  *out = op;
  return ABX_OK;
}

extern "C" int abx_fmm_stats(abx_operator *op, int64_t *m2l_pairs, int64_t *matrices,
                             int64_t *leaves, double *plan_seconds) {
  ABX_REQUIRE(op && op->kind == 2 && op->fmm, ABX_ERR_INVALID, "not an FMM operator");
  if (m2l_pairs) *m2l_pairs = op->fmm->n_m2l;
  if (matrices) *matrices = op->fmm->nmat;
  if (leaves) *leaves = op->fmm->nleaves;
  if (plan_seconds) *plan_seconds = op->fmm->build_s;
  return ABX_OK;
}

extern "C" int abx_fmm_set_wait_limit(abx_operator *op, double seconds, int drop_one_arrive) {
  ABX_REQUIRE(op && op->kind == 2 && op->fmm, ABX_ERR_INVALID, "not an FMM operator");
  ABX_REQUIRE(seconds > 0.0 && seconds <= 60.0, ABX_ERR_INVALID,
              "wait limit must be in (0, 60] seconds");
  op->fmm->wait_limit_s = seconds;
  op->fmm->drop_arrive = drop_one_arrive ? 1 : 0;
  return ABX_OK;
}
