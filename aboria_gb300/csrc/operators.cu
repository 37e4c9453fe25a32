// Kernel operators: create_sparse_operator / create_dense_operator and K*b.
//
// Reference: MatrixReplacement (src/Operators.h:75-281) with the Eigen product
// specialisation generic_product_impl::scaleAndAddTo
// (src/detail/Operators.h:207-229), which zero-initialises the destination and
// calls KernelX::evaluate.  The dense kernel restates KernelDense::evaluate
// (src/Kernels.h:212-239): for each row i, c_i = sum over j of f(a_i, b_j) * b_j.
// The reference adds the columns in order; here a thread owns a row and walks a
// chunk of them in order, 256 staged in shared memory at a time, and the chunks, as
// many as the rows leave SMs idle (dense_chunks), are added in order.  So the
// roundings are not the reference's and may differ between GPUs of other sizes.
#include <cmath>

#include "common.cuh"
#include "fix64.cuh"
#include "handles.cuh"

namespace abx {
namespace {

constexpr int DT = 256;  // rows per CTA = staged columns per tile

struct DenseParams {
  int dim, kind;
  double p0;
  float p0f, c_exp2;
  int64_t nr, nc;
  const double *rpos, *cpos;  // SoA storage order
  const double *b;
  const double *s_row, *s_col;
  double *c;
  double origin[3];
};

template <int KIND> __device__ __forceinline__ double dk64(double d2, double p0, double si,
                                                           double sj) {
  if (KIND == ABX_K_CONST) return p0;
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return exp(-d2 * p0);
  if (KIND == ABX_K_WENDLAND_C2) {
    const double q = sqrt(d2) * p0;
    if (q >= 1.0) return 0.0;
    const double t = 1.0 - q;
    const double t2 = t * t;
    return t2 * t2 * (4.0 * q + 1.0);
  }
  if (KIND == ABX_K_LAPLACE) return 1.0 / (sqrt(d2) + p0);
  if (KIND == ABX_K_MULTIQUADRIC) return sqrt(d2 + p0);
  if (KIND == ABX_K_SCALAR_SUM) return si + sj;
  return 0.0;
}

// Hardware base-2 exponential (MUFU, ~2 ulp), flush-to-zero: the kernel
// weights it serves are negligible long before 2^-126.
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <int KIND> __device__ __forceinline__ float dk32(float d2, float p0f, float c_exp2) {
  if (KIND == ABX_K_CONST) return p0f;
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) return ex2_approx(d2 * c_exp2);
  if (KIND == ABX_K_WENDLAND_C2) {
    const float q = d2 * rsqrtf(fmaxf(d2, 1e-36f)) * p0f;
    const float t = fmaxf(1.0f - q, 0.0f);
    const float t2 = t * t;
    return t2 * t2 * fmaf(4.0f, q, 1.0f);
  }
  if (KIND == ABX_K_LAPLACE) return __fdividef(1.0f, d2 * rsqrtf(fmaxf(d2, 1e-36f)) + p0f);
  if (KIND == ABX_K_MULTIQUADRIC) {
    const float a = d2 + p0f;
    return a * rsqrtf(fmaxf(a, 1e-36f));
  }
  return 0.f;
}

// `F` (may be null): leave at once where k_dense_fix has done the product.  Constant
// and scalar-sum kernels, which have no fixed-point values, come here only.  Column
// chunks (blockIdx.y) as in k_dense_fix: with one CTA per 256 rows, 460 x 1484
// took 2.0 ms, the latency of 1,484 values one after the other; with
// chunks 124 us.
template <int KIND>
__device__ __forceinline__ void dense_rows_fp64(const DenseParams &P, int64_t chunk_cols,
                                                double *__restrict__ partial) {
  __shared__ double sx[DT], sy[DT], sz[DT], sb[DT], ss[DT];
  const int64_t i = (int64_t)blockIdx.x * DT + threadIdx.x;
  const bool act = i < P.nr;
  double x0 = 0.0, x1 = 0.0, x2 = 0.0;
  if (act) {
    x0 = P.rpos[i];
    if (P.dim > 1) x1 = P.rpos[P.nr + i];
    if (P.dim > 2) x2 = P.rpos[2 * P.nr + i];
  }
  const double si = (KIND == ABX_K_SCALAR_SUM && act) ? P.s_row[i] : 0.0;
  double acc = 0.0;
  const int64_t c0 = (int64_t)blockIdx.y * chunk_cols;
  const int64_t c1 = c0 + chunk_cols < P.nc ? c0 + chunk_cols : P.nc;
  for (int64_t t = c0; t < c1; t += DT) {
    const int64_t j = t + threadIdx.x;
    if (j < c1) {
      sx[threadIdx.x] = P.cpos[j];
      sy[threadIdx.x] = P.dim > 1 ? P.cpos[P.nc + j] : 0.0;
      sz[threadIdx.x] = P.dim > 2 ? P.cpos[2 * P.nc + j] : 0.0;
      sb[threadIdx.x] = P.b[j];
      ss[threadIdx.x] = (KIND == ABX_K_SCALAR_SUM) ? P.s_col[j] : 0.0;
    }
    __syncthreads();
    const int nt = (int)((c1 - t) < DT ? (c1 - t) : DT);
    for (int jj = 0; jj < nt; ++jj) {
      // sum of squares in dimension order (0 + dx0^2 is exact)
      const double dx0 = __dsub_rn(sx[jj], x0);
      double d2 = __dmul_rn(dx0, dx0);
      if (P.dim > 1) {
        const double dx1 = __dsub_rn(sy[jj], x1);
        d2 = __dadd_rn(d2, __dmul_rn(dx1, dx1));
      }
      if (P.dim > 2) {
        const double dx2 = __dsub_rn(sz[jj], x2);
        d2 = __dadd_rn(d2, __dmul_rn(dx2, dx2));
      }
      acc = __dadd_rn(acc, __dmul_rn(dk64<KIND>(d2, P.p0, si, ss[jj]), sb[jj]));
    }
    __syncthreads();
  }
  if (!act) return;
  if (partial) partial[(int64_t)blockIdx.y * P.nr + i] = acc;
  else P.c[i] = acc;
}
struct DenseFix;
__device__ bool dense_fix_done(const DenseFix *F);
template <int KIND>
__global__ void __launch_bounds__(DT) k_dense_fp64(DenseParams P, const DenseFix *F,
                                                   int64_t chunk_cols, double *__restrict__ partial) {
  if (F && dense_fix_done(F)) return;
  dense_rows_fp64<KIND>(P, chunk_cols, partial);
}

// Kernel values of two pairs: packed FP32x2 where the formula allows.
template <int KIND> __device__ __forceinline__ float2 dk32x2(float2 dd, float p0f, float c_exp2) {
  if (KIND == ABX_K_GAUSSIAN || KIND == ABX_K_COMPACT_GAUSSIAN) {
    const float2 e = __fmul2_rn(dd, make_float2(c_exp2, c_exp2));
    return make_float2(ex2_approx(e.x), ex2_approx(e.y));
  }
  return make_float2(dk32<KIND>(dd.x, p0f, c_exp2), dk32<KIND>(dd.y, p0f, c_exp2));
}

// Mixed precision: FP32 offsets from the column domain centre, FP32 kernel
// values, one row per thread against two columns per packed FP32x2
// instruction; each staged tile of DT columns is summed in FP32 and tiles are
// added in FP64.  blockIdx.y selects a chunk of chunk_cols columns, so that
// small row counts still fill the GPU; with more than one chunk each CTA
// writes its row sums to partial[chunk][row] and k_dense_reduce adds the
// chunks in order (deterministic).  Columns are staged as pairs, pp[2h] = (x_a, x_b, y_a, y_b),
// pp[2h+1] = (z_a, z_b, b_a, b_b); an odd tail is paired with a far-away
// column of weight 0 (finite for every kernel).
template <int KIND>
__global__ void __launch_bounds__(DT) k_dense_mixed(DenseParams P, int64_t chunk_cols,
                                                    double *__restrict__ partial) {
  __shared__ float4 pp[DT];
  const int64_t i = (int64_t)blockIdx.x * DT + threadIdx.x;
  const bool act = i < P.nr;
  float x0 = 0.f, x1 = 0.f, x2 = 0.f;
  if (act) {
    x0 = (float)(P.rpos[i] - P.origin[0]);
    if (P.dim > 1) x1 = (float)(P.rpos[P.nr + i] - P.origin[1]);
    if (P.dim > 2) x2 = (float)(P.rpos[2 * P.nr + i] - P.origin[2]);
  }
  const float2 nqx = make_float2(-x0, -x0), nqy = make_float2(-x1, -x1), nqz = make_float2(-x2, -x2);
  double acc = 0.0;
  const int64_t c0 = (int64_t)blockIdx.y * chunk_cols;
  const int64_t c1 = c0 + chunk_cols < P.nc ? c0 + chunk_cols : P.nc;
  for (int64_t t = c0; t < c1; t += DT) {
    const int64_t j = t + threadIdx.x;
    float x = 1e4f, y = 1e4f, z = 1e4f, w = 0.f;
    if (j < c1) {
      x = (float)(P.cpos[j] - P.origin[0]);
      y = P.dim > 1 ? (float)(P.cpos[P.nc + j] - P.origin[1]) : 0.f;
      z = P.dim > 2 ? (float)(P.cpos[2 * P.nc + j] - P.origin[2]) : 0.f;
      w = (float)P.b[j];
    }
    float *pf = reinterpret_cast<float *>(&pp[2 * (threadIdx.x >> 1)]);
    const int o = threadIdx.x & 1;
    pf[o] = x;
    pf[2 + o] = y;
    pf[4 + o] = z;
    pf[6 + o] = w;
    __syncthreads();
    const int nt = (int)((c1 - t) < DT ? (c1 - t) : DT);
    const int npair = (nt + 1) >> 1;
    float2 a2 = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int h = 0; h < npair; ++h) {
      const float4 A = pp[2 * h], B = pp[2 * h + 1];
      const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nqx);
      const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nqy);
      const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nqz);
      float2 dd = __fmul2_rn(dx, dx);
      dd = __ffma2_rn(dy, dy, dd);
      dd = __ffma2_rn(dz, dz, dd);
      a2 = __ffma2_rn(dk32x2<KIND>(dd, P.p0f, P.c_exp2), make_float2(B.z, B.w), a2);
    }
    acc += (double)(a2.x + a2.y);
    __syncthreads();
  }
  if (act) {
    if (partial) partial[(int64_t)blockIdx.y * P.nr + i] = acc;
    else P.c[i] = acc;
  }
}

// ---------------------------------------------------- FP64 on integer units ---
// The default (FP64) dense product, for kernels and sizes that fix64.cuh
// covers: every pair costs one FP64 multiply-add instead of ~30 FP64
// operations.  Bounds: integer ALU (about 50 operations a pair at 62 a clock
// and SM) next to the one FP64 multiply-add (at 1.8).  Rows stay one a
// thread; columns, as fixed-point coordinates with their weights, are staged
// 256 at a time and read by broadcast; column chunks (blockIdx.y) fill the GPU
// when there are few rows and are added in order.  N = 32,768 x 30,011
// Gaussian: 57.6 -> 4.4 ms (error against 64 bits 5.2e-15 -> 1.2e-15).
//
// The unit of the fixed-point coordinates follows from the diagonal of both
// sets' bounding box, which k_dense_range finds on the device.  Where
// make_unit does not allow the integer path, or a coordinate is not finite,
// k_dense_fix leaves at once and k_dense_fp64 does the work; otherwise
// k_dense_fp64 leaves at once.
struct DenseFix {
  fx::Unit U;
  unsigned long long range[6];  // ordered bits: max of x_d, then max of -x_d
};
struct alignas(32) FixCol {
  long long x, y, z;
  double b;
};

__device__ bool dense_fix_done(const DenseFix *F) { return F->U.ok != 0; }

__device__ __forceinline__ unsigned long long ordered_bits(unsigned long long u) {
  return (u >> 63) ? ~u : u | 0x8000000000000000ull;
}
__device__ __forceinline__ double from_ordered(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k & 0x7fffffffffffffffull : ~k));
}

// Maxima of x_d and -x_d over every step-th point of two sets from `first` on, for the
// whole CTA, to `out` (thread 0), on the bits in an order-preserving form: a NaN of
// either sign sorts beyond the infinities and is caught with them (floating-point
// negation and comparison would lose its sign).
template <class Out>
__device__ __forceinline__ void dense_range(const DenseParams &P, int64_t first, int64_t step, Out out) {
  __shared__ unsigned long long red[DT / 32];
  for (int d = 0; d < P.dim; ++d) {
    unsigned long long hi = 0, lo = 0;
    for (int64_t i = first + threadIdx.x; i < P.nr + P.nc; i += step) {
      const unsigned long long u = (unsigned long long)__double_as_longlong(
          i < P.nr ? P.rpos[d * P.nr + i] : P.cpos[d * P.nc + (i - P.nr)]);
      hi = max(hi, ordered_bits(u));
      lo = max(lo, ordered_bits(u ^ 0x8000000000000000ull));
    }
    for (int s = 0; s < 2; ++s) {
      unsigned long long v = s ? lo : hi;
      for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < DT / 32; ++w) v = max(v, red[w]);
        out(3 * s + d, v);
      }
      __syncthreads();
    }
  }
}
__global__ void __launch_bounds__(DT) k_dense_range(DenseParams P, DenseFix *__restrict__ F) {
  dense_range(P, (int64_t)blockIdx.x * DT, (int64_t)gridDim.x * DT,
              [&](int k, unsigned long long v) { atomicMax(&F->range[k], v); });
}

// The kernel's unit from the ranges (one thread's work, done by every CTA that
// needs it before its columns).
template <int KIND> __device__ fx::Unit dense_unit(const DenseParams &P,
                                                   const unsigned long long *range) {
  double ext2 = 0.0;
  bool ok = true;
  for (int d = 0; d < P.dim; ++d) {
    const double hi = from_ordered(range[d]), lo = -from_ordered(range[3 + d]);
    ok = ok && isfinite(hi) && isfinite(lo);
    ext2 += (hi - lo) * (hi - lo);
  }
  fx::Unit U = fx::make_unit<KIND>(P.p0, ext2 > 0.0 ? sqrt(ext2) : 1e-30);
  U.ok = U.ok && ok;
  return U;
}

template <int KIND>
__device__ __forceinline__ FixCol fix_col(const DenseParams &P, const fx::Unit &U, int64_t j) {
  FixCol c;
  c.x = fx::fixed<KIND>(P.cpos[j], U);
  c.y = P.dim > 1 ? fx::fixed<KIND>(P.cpos[P.nc + j], U) : 0;
  c.z = P.dim > 2 ? fx::fixed<KIND>(P.cpos[2 * P.nc + j], U) : 0;
  c.b = P.b[j];
  return c;
}

template <int KIND>
__global__ void __launch_bounds__(DT) k_dense_prep(DenseParams P, DenseFix *__restrict__ Fg,
                                                   FixCol *__restrict__ cols) {
  __shared__ fx::Unit U;
  if (threadIdx.x == 0) {
    U = dense_unit<KIND>(P, Fg->range);
    if (blockIdx.x == 0) Fg->U = U;
  }
  __syncthreads();
  const int64_t j = (int64_t)blockIdx.x * DT + threadIdx.x;
  if (U.ok && j < P.nc) cols[j] = fix_col<KIND>(P, U, j);
}

// `cols` null: the columns are put into fixed point as they are staged.
template <int KIND, int DIM>
__device__ __forceinline__ void dense_rows_fix(const DenseParams &P, const fx::Unit &U,
                                               const FixCol *__restrict__ cols, int64_t chunk_cols,
                                               double *__restrict__ partial) {
  __shared__ FixCol sc[DT];
  __shared__ fx::u64 tab[fx::EXP_TAB];
  if (KIND == ABX_K_GAUSSIAN) tab[threadIdx.x] = fx::exp_table.v[threadIdx.x];
  const fx::Consts C = fx::consts(U, 1.0 / P.p0);
  const int64_t i = (int64_t)blockIdx.x * DT + threadIdx.x;
  const bool act = i < P.nr;
  long long x = 0, y = 0, z = 0;
  if (act) {
    x = fx::biased(fx::fixed<KIND>(P.rpos[i], U));
    if (DIM > 1) y = fx::biased(fx::fixed<KIND>(P.rpos[P.nr + i], U));
    if (DIM > 2) z = fx::biased(fx::fixed<KIND>(P.rpos[2 * P.nr + i], U));
  }
  double acc = 0.0;
  const int64_t c0 = (int64_t)blockIdx.y * chunk_cols;
  const int64_t c1 = c0 + chunk_cols < P.nc ? c0 + chunk_cols : P.nc;
  for (int64_t t = c0; t < c1; t += DT) {
    __syncthreads();
    if (t + threadIdx.x < c1)
      sc[threadIdx.x] = cols ? cols[t + threadIdx.x] : fix_col<KIND>(P, U, t + threadIdx.x);
    __syncthreads();
    const int nt = (int)((c1 - t) < DT ? (c1 - t) : DT);
#pragma unroll 2
    for (int jj = 0; jj < nt; ++jj) {
      const FixCol q = sc[jj];
      bool near;
      double v = fx::value<KIND>(fx::diff(q.x, x), fx::diff(q.y, y), fx::diff(q.z, z), DIM, C, tab,
                                 near);
      if (KIND == ABX_K_LAPLACE && near && act) {
        double a[DIM], b[DIM];
        bool same = true;  // two points in one place have the value at distance 0
        for (int d = 0; d < DIM; ++d) {
          a[d] = P.cpos[d * P.nc + t + jj];
          b[d] = P.rpos[d * P.nr + i];
          same = same && __double_as_longlong(a[d]) == __double_as_longlong(b[d]);
        }
        if (!same) {
          double d2 = 0.0;
          for (int d = 0; d < DIM; ++d) {
            const double dx = a[d] - b[d];
            d2 = __dadd_rn(d2, __dmul_rn(dx, dx));
          }
          v = dk64<KIND>(d2, P.p0, 0.0, 0.0);
        }
      }
      acc = fma(v, q.b, acc);
    }
  }
  if (act) {
    if (partial) partial[(int64_t)blockIdx.y * P.nr + i] = acc;
    else P.c[i] = acc;
  }
}
template <int KIND, int DIM>
__global__ void __launch_bounds__(DT) k_dense_fix(DenseParams P, const DenseFix *__restrict__ Fg,
                                                  const FixCol *__restrict__ cols,
                                                  int64_t chunk_cols, double *__restrict__ partial) {
  if (!Fg->U.ok) return;
  const fx::Unit U = Fg->U;
  dense_rows_fix<KIND, DIM>(P, U, cols, chunk_cols, partial);
}

// The whole product of two small sets in one launch: every CTA goes over all points
// for the ranges (L2 holds them) and puts its own columns into fixed point, or takes
// the FP64 formula.  Four launches, of which one does the work, are what such a
// product took: 1 x 1 37 us, 25 so; 300 x 300 Gaussian 101, 84.
constexpr int64_t DENSE_SMALL = 2048;  // points
template <int KIND, int DIM>
__global__ void __launch_bounds__(DT) k_dense_small(DenseParams P, int64_t chunk_cols,
                                                    double *__restrict__ partial) {
  __shared__ unsigned long long range[6];
  __shared__ fx::Unit U;
  dense_range(P, 0, DT, [&](int k, unsigned long long v) { range[k] = v; });
  if (threadIdx.x == 0) U = dense_unit<KIND>(P, range);
  __syncthreads();
  if (U.ok)
    dense_rows_fix<KIND, DIM>(P, U, nullptr, chunk_cols, partial);
  else
    dense_rows_fp64<KIND>(P, chunk_cols, partial);
}

__global__ void k_dense_reduce(const double *__restrict__ partial, int64_t nr, int chunks,
                               double *__restrict__ c) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nr) return;
  double s = 0.0;
  for (int k = 0; k < chunks; ++k) s += partial[(int64_t)k * nr + i];
  c[i] = s;
}

// Columns in chunks of whole tiles when the rows alone give fewer than about
// per_sm CTAs per SM; returns the number of chunks, at least 1.
int dense_chunks(abx_context *ctx, int64_t nc, unsigned blocks, int per_sm, int64_t &chunk_cols) {
  const int64_t tiles = (nc + DT - 1) / DT;
  const int64_t want = (per_sm * (int64_t)std::max(ctx->num_sms, 1) + blocks - 1) / blocks;
  const int chunks = (int)std::max<int64_t>(1, std::min<int64_t>(want, std::min<int64_t>(tiles, 65535)));
  // no columns: one chunk that writes zeros
  chunk_cols = tiles > 0 ? ((tiles + chunks - 1) / chunks) * DT : DT;
  return tiles > 0 ? (int)((nc + chunk_cols - 1) / chunk_cols) : 1;
}

// Room for an FP64 product of nr x nc.
size_t dense_room(abx_context *ctx, int64_t nr, int64_t nc) {
  int64_t chunk_cols;
  const int used = dense_chunks(ctx, nc, ceil_div(nr, DT), 16, chunk_cols);
  return sizeof(DenseFix) / 8 + 4 + (sizeof(FixCol) / 8) * (size_t)nc +
         (used > 1 ? (size_t)used * nr : 0);
}
int dense_reserve(abx_context *ctx, int64_t nr, int64_t nc, abx_operator *op) {
  return op->partial.reserve(dense_room(ctx, nr, nc));
}

template <int KIND>
int launch_dense_fix(abx_context *ctx, const DenseParams &P, abx_operator *op) {
  cudaStream_t s = ctx->stream;
  const unsigned blocks = ceil_div(P.nr, DT);
  int64_t chunk_cols;
  const int used = dense_chunks(ctx, P.nc, blocks, 16, chunk_cols);
  // one buffer: the unit, the columns, the chunks' row sums
  const size_t nf = sizeof(DenseFix) / 8 + 4, nb = (sizeof(FixCol) / 8) * (size_t)P.nc;
  ABX_TRY(dense_reserve(ctx, P.nr, P.nc, op));
  DenseFix *F = reinterpret_cast<DenseFix *>(op->partial.ptr);
  FixCol *cols = reinterpret_cast<FixCol *>(op->partial.ptr + (nf / 4) * 4);
  double *partial = used > 1 ? op->partial.ptr + (nf / 4) * 4 + nb : nullptr;
  const dim3 grid(blocks, used);
  if (P.nr + P.nc <= DENSE_SMALL) {
    if (P.dim == 3)
      k_dense_small<KIND, 3><<<grid, DT, 0, s>>>(P, chunk_cols, partial);
    else if (P.dim == 2)
      k_dense_small<KIND, 2><<<grid, DT, 0, s>>>(P, chunk_cols, partial);
    else
      k_dense_small<KIND, 1><<<grid, DT, 0, s>>>(P, chunk_cols, partial);
    if (partial) k_dense_reduce<<<ceil_div(P.nr, 256), 256, 0, s>>>(partial, P.nr, used, P.c);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  ABX_CHECK_CUDA(cudaMemsetAsync(F, 0, sizeof(DenseFix), s));
  const unsigned rb = std::min(ceil_div(P.nr + P.nc, DT), 2u * (unsigned)std::max(ctx->num_sms, 1));
  k_dense_range<<<rb, DT, 0, s>>>(P, F);
  k_dense_prep<KIND><<<std::max(1u, ceil_div(P.nc, DT)), DT, 0, s>>>(P, F, cols);
  if (P.dim == 3)
    k_dense_fix<KIND, 3><<<grid, DT, 0, s>>>(P, F, cols, chunk_cols, partial);
  else if (P.dim == 2)
    k_dense_fix<KIND, 2><<<grid, DT, 0, s>>>(P, F, cols, chunk_cols, partial);
  else
    k_dense_fix<KIND, 1><<<grid, DT, 0, s>>>(P, F, cols, chunk_cols, partial);
  k_dense_fp64<KIND><<<grid, DT, 0, s>>>(P, F, chunk_cols, partial);
  if (partial) k_dense_reduce<<<ceil_div(P.nr, 256), 256, 0, s>>>(partial, P.nr, used, P.c);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

template <int KIND>
int launch_dense(abx_context *ctx, const DenseParams &P, bool mixed, abx_operator *op) {
  const unsigned blocks = ceil_div(P.nr, DT);
  if (mixed && KIND != ABX_K_SCALAR_SUM) {
    int64_t chunk_cols;
    const int used = dense_chunks(ctx, P.nc, blocks, 32, chunk_cols);
    double *partial = nullptr;
    if (used > 1) {
      ABX_TRY(op->partial.reserve((size_t)used * P.nr));
      partial = op->partial.ptr;
    }
    k_dense_mixed<KIND><<<dim3(blocks, std::max(used, 1)), DT, 0, ctx->stream>>>(P, chunk_cols,
                                                                               partial);
    if (partial)
      k_dense_reduce<<<ceil_div(P.nr, 256), 256, 0, ctx->stream>>>(partial, P.nr, used, P.c);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  if (op->partial.cap < dense_room(ctx, P.nr, P.nc) && stream_capturing(ctx->stream)) {
    // no room, and none to be had: one CTA walks all columns
    k_dense_fp64<KIND><<<blocks, DT, 0, ctx->stream>>>(P, nullptr, P.nc, nullptr);
    ABX_CHECK_CUDA(cudaGetLastError());
    return ABX_OK;
  }
  if constexpr (KIND != ABX_K_CONST && KIND != ABX_K_SCALAR_SUM) {
    // the two Gaussians share one instantiation
    if (P.nc > 0)
      return launch_dense_fix<KIND == ABX_K_COMPACT_GAUSSIAN ? ABX_K_GAUSSIAN : KIND>(ctx, P, op);
  }
  int64_t chunk_cols;
  const int used = dense_chunks(ctx, P.nc, blocks, 16, chunk_cols);
  ABX_TRY(dense_reserve(ctx, P.nr, P.nc, op));
  double *partial = used > 1 ? op->partial.ptr : nullptr;
  k_dense_fp64<KIND><<<dim3(blocks, used), DT, 0, ctx->stream>>>(P, nullptr, chunk_cols, partial);
  if (partial)
    k_dense_reduce<<<ceil_div(P.nr, 256), 256, 0, ctx->stream>>>(partial, P.nr, used, P.c);
  ABX_CHECK_CUDA(cudaGetLastError());
  return ABX_OK;
}

}  // namespace

int dense_matvec_device(abx_operator *op, const double *b, double *c) {
  abx_context *ctx = op->rows->ctx;
  DenseParams P{};
  P.dim = op->rows->dim;
  P.kind = op->k.kind;
  P.p0 = op->k.p[0];
  P.p0f = (float)op->k.p[0];
  P.c_exp2 = (float)(-op->k.p[0] * 1.4426950408889634);
  P.nr = op->rows->n;
  P.nc = op->cols->n;
  P.rpos = op->rows->pos.ptr;
  P.cpos = op->cols->pos.ptr;
  P.b = b;
  P.c = c;
  if (P.kind == ABX_K_SCALAR_SUM) {
    ABX_REQUIRE(op->rows->has_scalar && op->cols->has_scalar, ABX_ERR_STATE,
                "ABX_K_SCALAR_SUM needs a scalar column on both particle sets");
    P.s_row = op->rows->scalar.ptr;
    P.s_col = op->cols->scalar.ptr;
  }
  // FP32 coordinates are taken relative to the column domain centre when a
  // domain is set, else to the origin.
  for (int d = 0; d < 3; ++d) P.origin[d] = 0.0;
  if (op->cols->domain_set)
    for (int d = 0; d < P.dim; ++d)
      P.origin[d] = 0.5 * (op->cols->grid.lo[d] + op->cols->grid.hi[d]);
  if (P.nr == 0) return ABX_OK;
  const bool mixed = op->precision == ABX_PREC_MIXED;
  switch (P.kind) {
  case ABX_K_CONST: return launch_dense<ABX_K_CONST>(ctx, P, mixed, op);
  case ABX_K_GAUSSIAN: return launch_dense<ABX_K_GAUSSIAN>(ctx, P, mixed, op);
  case ABX_K_WENDLAND_C2: return launch_dense<ABX_K_WENDLAND_C2>(ctx, P, mixed, op);
  case ABX_K_COMPACT_GAUSSIAN: return launch_dense<ABX_K_COMPACT_GAUSSIAN>(ctx, P, mixed, op);
  case ABX_K_LAPLACE: return launch_dense<ABX_K_LAPLACE>(ctx, P, mixed, op);
  case ABX_K_MULTIQUADRIC: return launch_dense<ABX_K_MULTIQUADRIC>(ctx, P, mixed, op);
  case ABX_K_SCALAR_SUM: return launch_dense<ABX_K_SCALAR_SUM>(ctx, P, false, op);
  }
  set_error("unknown kernel kind %d", P.kind);
  return ABX_ERR_INVALID;
}

}  // namespace abx

using namespace abx;

extern "C" {

static int check_kernel(const abx_kernel *k) {
  ABX_REQUIRE(k, ABX_ERR_INVALID, "null kernel descriptor");
  ABX_REQUIRE(k->kind >= ABX_K_CONST && k->kind <= ABX_K_SCALAR_SUM, ABX_ERR_INVALID,
              "unknown kernel kind %d", k->kind);
  return ABX_OK;
}

int abx_create_sparse_operator(abx_particles *rows, abx_particles *cols, double radius,
                               const abx_kernel *k, abx_operator **out) {
  ABX_REQUIRE(rows && cols && out, ABX_ERR_INVALID, "null argument");
  ABX_TRY(check_kernel(k));
  ABX_REQUIRE(rows->ctx == cols->ctx, ABX_ERR_INVALID, "particle sets on different contexts");
  ABX_REQUIRE(rows->dim == cols->dim, ABX_ERR_INVALID, "dimension mismatch");
  ABX_REQUIRE(cols->searchable, ABX_ERR_STATE,
              "init_neighbour_search not called on the column particle set");
  ABX_REQUIRE(radius >= 0 && std::isfinite(radius), ABX_ERR_INVALID, "invalid radius");
  ABX_TRY(ctx_activate(rows->ctx));
  abx_operator *op = new abx_operator();
  op->kind = 0;
  op->rows = rows;
  op->cols = cols;
  op->radius = radius;
  op->k = *k;
  int st = pair_layout_build(op);
  if (st != ABX_OK) {
    if (op->pairs) pair_layout_free(op->pairs);
    delete op;
    return st;
  }
  particles_retain(rows);
  particles_retain(cols);
  *out = op;
  return ABX_OK;
}

int abx_create_dense_operator(abx_particles *rows, abx_particles *cols, const abx_kernel *k,
                              abx_operator **out) {
  ABX_REQUIRE(rows && cols && out, ABX_ERR_INVALID, "null argument");
  ABX_TRY(check_kernel(k));
  ABX_REQUIRE(rows->ctx == cols->ctx, ABX_ERR_INVALID, "particle sets on different contexts");
  ABX_REQUIRE(rows->dim == cols->dim, ABX_ERR_INVALID, "dimension mismatch");
  abx_operator *op = new abx_operator();
  op->kind = 1;
  op->rows = rows;
  op->cols = cols;
  op->k = *k;
  particles_retain(rows);
  particles_retain(cols);
  *out = op;
  return ABX_OK;
}

int abx_operator_destroy(abx_operator *op) {
  if (!op) return ABX_OK;
  abx_particles *rows = op->rows, *cols = op->cols;
  cudaSetDevice(rows->ctx->device);
  cudaStreamSynchronize(rows->ctx->stream);
  if (op->pairs) pair_layout_free(op->pairs);
  if (op->fmm) fmm_plan_free(op->fmm);
  delete op;
  particles_release(rows);
  particles_release(cols);
  return ABX_OK;
}

int abx_operator_set_precision(abx_operator *op, int mode) {
  ABX_REQUIRE(op, ABX_ERR_INVALID, "null operator");
  ABX_REQUIRE(mode == ABX_PREC_FP64 || mode == ABX_PREC_MIXED, ABX_ERR_INVALID,
              "unknown precision mode %d", mode);
  // the buffers of an FP64 product, so that the first one allocates nothing
  if (mode == ABX_PREC_FP64 && op->kind == 1 && op->rows->n > 0) {
    ABX_TRY(ctx_activate(op->rows->ctx));
    ABX_TRY(dense_reserve(op->rows->ctx, op->rows->n, op->cols->n, op));
  }
  if (mode == ABX_PREC_FP64 && op->fmm) {
    ABX_TRY(ctx_activate(op->rows->ctx));
    ABX_TRY(fmm_plan_prepare(op->fmm, op->rows->n, op->rows->ctx->stream));
  }
  op->precision = mode;
  return ABX_OK;
}

int64_t abx_operator_rows(const abx_operator *op) { return op ? op->rows->n : -1; }
int64_t abx_operator_cols(const abx_operator *op) { return op ? op->cols->n : -1; }

int abx_operator_matvec(abx_operator *op, const double *b, double *c) {
  ABX_REQUIRE(op, ABX_ERR_INVALID, "null operator");
  const int64_t nr = op->rows->n, nc = op->cols->n;
  ABX_REQUIRE((b || nc == 0) && (c || nr == 0), ABX_ERR_INVALID, "null vector");
  abx_context *ctx = op->rows->ctx;
  ABX_TRY(ctx_activate(ctx));
  if (op->kind == 0)
    ABX_REQUIRE(op->cols->searchable, ABX_ERR_STATE,
                "init_neighbour_search not called on the column particle set");
  const void *bd;
  void *cd;
  ABX_TRY(op->stage_b.in(ctx, b, (size_t)nc * sizeof(double), &bd));
  ABX_TRY(op->stage_c.out(ctx, c, (size_t)nr * sizeof(double), &cd));
  if (op->kind == 0)
    ABX_TRY(sparse_matvec_device(op, (const double *)bd, (double *)cd));
  else if (op->kind == 1)
    ABX_TRY(dense_matvec_device(op, (const double *)bd, (double *)cd));
  else
    ABX_TRY(fmm_matvec_device(op, (const double *)bd, (double *)cd));
  ABX_TRY(op->stage_c.finish(ctx, c, (size_t)nr * sizeof(double)));
  return ABX_OK;
}

int abx_operator_last_stats(abx_operator *op, int64_t *candidates, int64_t *pairs) {
  ABX_REQUIRE(op, ABX_ERR_INVALID, "null operator");
  if (candidates) *candidates = op->last_candidates;
  if (pairs) *pairs = op->last_pairs;
  return ABX_OK;
}

}  // extern "C"
