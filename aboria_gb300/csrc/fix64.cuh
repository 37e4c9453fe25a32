// FP64-accurate kernel values from integer and FP32 arithmetic.
//
// GB300 issues 2 FP64 operations per clock and SM (measured 1.7-1.8) against
// 62 integer ALU operations, 115 FP32 FMAs and 25 32x32+64-bit multiply-adds of three
// registers (58 with a uniform operand), so one double-precision operation costs as
// much as about 32 integer ones.
// A pair's kernel value takes ~30 of the former (distance 6-8, sqrt or exp
// 10-20, the rest the polynomial and the product); here everything but the
// last multiply-add into the row's FP64 sum runs on the integer pipe:
//
//  * coordinates are 64-bit fixed point modulo 2^64, X = x f in a unit 2^-k
//    (to_fixed): differences that fit in 63 bits are exact whatever wrapped on
//    the way.  f is a power of two, so that a double's bits are shifted and
//    not rounded down to the unit, or, where that saves the pair a product,
//    the kernel's own scale: sqrt(p0 log2(e)) for the Gaussian, p0 for the
//    Wendland kernel, held to 100 bits (Unit);
//  * each difference is split as h 2^32 + l with a signed low half; h^2 and h l
//    are summed exactly; l^2, which is below the unit of the sum, counts for
//    Laplace and multiquadric values and Gaussians beyond 2^-255 (sq_acc, sq_low);
//  * sqrt starts from the hardware's FP32 reciprocal square root and takes
//    two corrections from exact integer residuals (sqrt60);
//  * 2^-t splits t into an exponent, an index of a 256-entry table and a rest
//    below 2^-8 whose Taylor series (ln 2 powers) is a Horner chain of
//    multiply-adds (exp2_neg).  Table-driven exponentials: P.T.P. Tang, ACM
//    TOMS 15 (1989).
//
// Relative errors, against 50 digits (tests/test_fix64.py): below 2^-52 for
// every value, 2^-54 rms, where the FP64 formulas have 2^-49.4 (Gaussian), 2^-51
// (1/(d + p0)) and 2^-51.5 (sqrt(d^2 + p0)) at worst and about 2^-53 rms, the
// Gaussian 2^-52; a Wendland value near its cut-off keeps 6 bits more than in
// FP64.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace abx {
namespace fx {

typedef uint64_t u64;
typedef int64_t i64;
typedef uint32_t u32;

FX_HD u32 hi32(u64 a) { return (u32)(a >> 32); }

// a b / 2^64 to within 1 unit for a, b <= 2^63: the low x low product is left
// out and the constant makes up for it and for the floor on average (the two
// middle products and the constant cannot overflow their sum).
FX_HD u64 mulhi63(u64 a, u64 b) {
  const u64 w = ((u64)(u32)a * hi32(b) + 0xc0000000ull) + (u64)hi32(a) * (u32)b;
  return (u64)hi32(a) * hi32(b) + (w >> 32);
}

FX_HD u64 bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  u64 u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
FX_HD double from_bits(u64 u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

FX_HD u64 mulhi64(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

// A positive factor f = F 2^-ef, F = fh 2^64 + fl with the top bit set.
struct Factor {
  u64 fh, fl;
  int ef;
};
// f = hi + lo, hi > 0 normal, |lo| <= ulp(hi)
FX_HD Factor make_factor(double hi, double lo) {
  const u64 u = bits_of(hi);
  const int e = (int)(u >> 52) - 1023;
  Factor F;
  F.fh = (u << 11) | (1ull << 63);
  F.fl = 0;
  F.ef = 127 - e;
  // lo in units of 2^(e - 127): 75 bits at most
  const double l1 = ldexp(lo, 63 - e);  // units of 2^64 F units
  const double w = floor(l1);
  F.fh += (u64)(i64)w;
  F.fl = (u64)ldexp(l1 - w, 63) << 1;
  return F;
}

// x f 2^k modulo 2^64, rounded to nearest; x finite.
FX_HD i64 to_fixed(double x, const Factor &F, int k) {
  const u64 u = bits_of(x);
  const int e = (int)((u >> 52) & 0x7ff);
  const u64 m = (u & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
  // |x| = m 2^(max(e, 1) - 1075); m F as three words
  const u64 p0 = m * F.fl, t = mulhi64(m, F.fl), a = m * F.fh;
  const u64 p1 = a + t, p2 = mulhi64(m, F.fh) + (p1 < a ? 1u : 0u);
  const int s = (e ? e : 1) - 1075 - F.ef + k;  // value = m F 2^s
  u64 v;
  if (s >= 64)
    v = 0;
  else if (s >= 0)
    v = p0 << s;
  else {
    const int r = -s, w = r >> 6, b = r & 63;
    const u64 lo = w == 0 ? p0 : w == 1 ? p1 : w == 2 ? p2 : 0;
    const u64 hi = w == 0 ? p1 : w == 1 ? p2 : 0;
    v = b ? (lo >> b) | (hi << (64 - b)) : lo;
    // the bit below the unit rounds
    const int rb = r - 1, rw = rb >> 6;
    const u64 below = rw == 0 ? p0 : rw == 1 ? p1 : rw == 2 ? p2 : 0;
    v += (below >> (rb & 63)) & 1;
  }
  return (i64)((u >> 63) ? 0 - v : v);
}

// A query's coordinate is kept shifted by 2^31 (biased), so that the upper half
// of a difference comes out rounded and its lower half as a signed number with
// the top bit inverted.
FX_HD i64 biased(i64 q) { return (i64)((u64)q - 0x80000000ull); }
FX_HD i64 diff(i64 x, i64 q_biased) { return (i64)((u64)x - (u64)q_biased); }
FX_HD int32_t low_of(i64 d) { return (int32_t)((u32)d ^ 0x80000000u); }
// Adds dx^2 to the split sum (d as diff() gives it).
FX_HD void sq_acc(i64 d, i64 &S, i64 &T) {
  const int32_t h = (int32_t)(d >> 32), l = low_of(d);
  S += (i64)h * h;
  T += (i64)h * l;
}
FX_HD u64 sq_low(i64 d) {
  const int32_t l = low_of(d);
  return (u64)((i64)l * l);
}
// The sum in units of u^2 2^64 for coordinates in units of u ...
FX_HD u64 sq_sum(i64 S, i64 T) { return (u64)S + (u64)(T >> 31); }
// ... and with BITS bits more (a sum below 2^(63 - BITS) of those units), for which
// the low parts' squares L (sq_low) count too.
template <int BITS> FX_HD u64 sq_sum_low(i64 S, i64 T, u64 L) {
  return ((u64)S << BITS) + (u64)((T + (i64)(L >> 33)) >> (31 - BITS));
}

FX_HD float rsqrt32(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / sqrtf(x);
#endif
}
FX_HD float rcp32(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
FX_HD int f2i(float x) {  // to nearest
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)lrintf(x);
#endif
}
FX_HD float fma32(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}
FX_HD int clz32(u32 x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

// sqrt(u 2^-60) in units of 2^-62 for u <= 3 2^60 (a root up to 1.74); the
// error is below 2^-60 for u >= 2^40.  q0 = the FP32 root as an integer (units
// 2^-30, relative error below 2^-21.5); with res = u - q0^2 exact, the
// correction is d - d^2 / (2 q0), d = res / (2 q0): D1 is d in units of 2^-50
// to FP32 accuracy, R1 what D1 leaves of res (exact), and the last FP32 term
// carries R1's and d^2's share.  u = 0 gives 0.
// SMALL: for any u, to 2^-60 / sqrt(u 2^-60) below 2^40.  The residual is shifted with
// rounding: the floor of -1 / 2^11 is -1, a correction by 2^11 / (2 q0), which for u
// below 2^22 was more than the root.
template <bool SMALL = false> FX_HD u64 sqrt60(u64 u) {
  const float uf = fma32((float)hi32(u), 4294967296.0f, (float)(u32)u);
  const float rs = rsqrt32(fmaxf(uf, 1.0f));
  const int q0 = f2i(uf * rs);
  const i64 res = (i64)u - (i64)q0 * q0;
  const float d1 = (float)(int32_t)((SMALL ? res + 1024 : res) >> 11) * (rs * 1073741824.0f);  // 2^11 2^20 / 2
  const int D1 = f2i(d1);
  const i64 R1 = (i64)((u64)res << 20) - (i64)q0 * (2 * D1);
  const float r1 = (float)(int32_t)(R1 >> 10);
  const float c = fma32(d1 * d1, -9.3132257461547852e-10f, r1) * (rs * 2097152.0f);
  const i64 low = (i64)D1 * 4096 + f2i(c);
  return (((u64)(u32)q0) << 32) + (u64)low;
}

// m 2^-s as a double for m in [2^61, 2^62], rounded to nearest.
FX_HD double make_double61(u64 m, int s) {
  const u64 r = (m + 256) >> 9;  // 53 bits; 2^53 carries into the exponent
  return from_bits(r + ((u64)(u32)(1083 - s) << 52));
}
FX_HD u32 funnel_l(u32 lo, u32 hi, int k) {  // upper word of (hi : lo) << k, 0 <= k < 32
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, k);
#else
  return k ? (hi << k) | (lo >> (32 - k)) : hi;
#endif
}
FX_HD u64 join(u32 hi, u32 lo) { return ((u64)hi << 32) | lo; }

// m * 2^-s as a double, rounded to nearest; m != 0, the result normal.
FX_HD double make_double(u64 m, int s) {
  const u32 h = hi32(m);
  const int z = h ? clz32(h) : 32 + clz32((u32)m);
  const u64 n = m << z;  // top bit set
  // 53 significant bits; the sum carries into the exponent where it rounds up
  const u64 r = (n >> 11) + ((n >> 10) & 1);
  return from_bits(r + ((u64)(1085 - z - s) << 52));
}

// ------------------------------------------------------------ exponential ---
constexpr int EXP_TAB = 256;
// 2^(-i/256) in units of 2^-63, from repeated integer square roots of 1/2 and
// their products: within 3.4 units (2^-61), and the same on every compiler;
// plus the half unit (512) that rounds a value to 53 bits, less what the
// products' floors leave out on average (3e-17 of the value).
struct ExpTable {
  u64 v[EXP_TAB];
};
constexpr ExpTable make_exp_table() {
  typedef unsigned __int128 u128;
  u64 root[8] = {};  // 2^(-2^k/256) in units of 2^-64
  u128 v = (u128)1 << 63;
  for (int k = 7; k >= 0; --k) {
    const u128 n = v << 64;
    u128 s = 0;
    for (int b = 63; b >= 0; --b) {
      const u128 t = s | ((u128)1 << b);
      if (t * t <= n) s = t;
    }
    v = s;
    root[k] = (u64)s;
  }
  ExpTable T{};
  for (int i = 0; i < EXP_TAB; ++i) {
    u128 p = (u128)1 << 64;
    for (int k = 0; k < 8; ++k)
      if ((i >> k) & 1) p = (p * root[k]) >> 64;
    T.v[i] = (u64)(p >> 1) + 305;
  }
  return T;
}
#ifdef __CUDACC__
static __device__ const ExpTable exp_table = make_exp_table();
#endif

// 2^-t for t in units of 2^-54 (t < 2^64: below 1024, the result normal below
// 1020), as a double.
// t = n + i/256 + g, g < 2^-8 as y = 2^8 g in units of 2^-63 (G);
// 1 - 2^-g = g (L1 - g (L2 - g (L3 - g (L4 - g L5)))), Lk = ln(2)^k / k!,
// the first neglected term below 2^-60.  Every Horner step is one 32x32+64
// multiply-add whose scale is folded into the constants:
// E = 2^64 (1 - 2^-g).
FX_HD double exp2_neg(u64 t, const u64 *tab) {
  const u32 th = hi32(t);
  const u64 G = (t & 0x3fffffffffffull) << 17;
  const int32_t g = (int32_t)hi32(G);  // y in units of 2^-31
  // n4 = -(L4 - g L5) in units of 2^-28; a3 = L3 - g(...) in units of 2^-35
  const int32_t n4 = (int32_t)((((i64)g * 2796) - ((i64)2581847 << 32)) >> 32);
  const int32_t a3 = (int32_t)((((i64)g * n4) + ((i64)1907106652 << 32)) >> 32);
  const int32_t ga3 = (int32_t)(((i64)g * a3) >> 32);  // y a3 in units of 2^-34
  // A2 = L2 - g a3 in units of 2^-50, A1 = L1 - g A2 in units of 2^-57
  const u64 A2 = (u64)((i64)ga3 * -256 + (i64)270471001806380ll);
  const u64 A1 = 99893036290645747ull - mulhi63(G, A2);
  const u64 E = mulhi63(G, A1);
  const u64 T = tab[(th >> 14) & (EXP_TAB - 1)];
  const u64 m = (T - mulhi63(T, E)) >> 10;  // 53 bits; 2^53 carries into the exponent
  return from_bits(m + ((u64)(1021u - (th >> 22)) << 52));
}

// ---------------------------------------------------------- kernel values ---
// Wendland C2 (1-q)^4 (4q+1) = t^4 (5 - 4t), t = 1 - q, for q^2 in units of
// 2^-60; 0 for q >= 1.  t is normalised, so that the value keeps its relative
// accuracy where t is small.
FX_HD double wendland(u64 q2) {
  if (q2 >= (1ull << 60)) return 0.0;
  const i64 td = (i64)(1ull << 62) - (i64)sqrt60<true>(q2);
  const u64 t = ((u64)td << 1) - (u64)(td >> 62);  // units of 2^-63, below 2^63
  const u32 th = hi32(t);
  if (td <= 0 || th == 0) return 0.0;  // t < 2^-31: the value is below 2^-121
  const int z = clz32(th) - 1;
  const u64 tn = t << z;                // in [2^62, 2^63)
  const u64 t2 = mulhi63(tn, tn) << 1;  // t^2 in units of 2^-63, >= 2^61
  const u64 t4 = mulhi63(t2, t2) << 1;  // t^4 in units of 2^-63, >= 2^59
  const u64 p = (5ull << 60) - (t >> 1);
  return make_double(mulhi63(t4, p), 59 + 4 * z);
}

// d >= 2^-7 R: the coordinates' rounding to 2^-62 R is below 2^-54 of d.  Closer
// pairs are left to the FP64 formula on the double coordinates.
FX_HD bool laplace_far(i64 S) { return S >= (i64)1 << 46; }

// |dx|^2 of a split sum with its low part U = sum l^2, normalised, for
// laplace_far pairs: the value is n 2^-62 2^-z R^2 with n in [2^62, 2^64) and z
// even, 0 <= z <= 14.
FX_HD u64 norm_d2(i64 S, i64 T, u64 U, int &z) {
  const u32 t0 = (u32)T << 1, low = hi32(U) + t0;  // the word below S's
  const u64 s = (u64)S + (u64)(T >> 31) + (low < t0 ? 1u : 0u);  // units of 2^-60
  const int k = clz32(hi32(s)) & ~1;  // at most 16
  z = k - 2;
  return join(funnel_l((u32)s, hi32(s), k), funnel_l(low, (u32)s, k));
}

// 1 / (d + p0) for laplace_far pairs: n, z as norm_d2 gives them, P0 = p0 / R in
// units of 2^-61 (p0 < R), R = 2^r.
FX_HD double laplace(u64 n, int z, u64 P0, int r) {
  // d = q 2^-62 2^(1 - z/2) R, q in [2^61, 2^62); a = d + p0 in units of 2^-61
  // (below 2^-55 of d), normalised to [2^62, 2^63)
  const u64 a = (sqrt60(n >> 4) >> (z >> 1)) + P0;
  const int y = clz32(hi32(a)) - 1;  // 2^54 <= a < 2^63
  const u64 A = join(funnel_l((u32)a, hi32(a), y), (u32)a << y);
  // reciprocal of A 2^-62 in [1, 2): FP32 seed, then 1 + e + e^2
  const u32 Y0 = (u32)f2i(rcp32((float)hi32(A) * 9.3132257461547852e-10f) * 1073741824.0f);
  const u64 w = (u64)(u32)A * Y0;
  const i64 er = (i64)((1ull << 60) - ((u64)hi32(A) * Y0 + (w >> 32)));
  const i64 es = er >> 20;
  const i64 e2 = er + ((es * es) >> 20);
  const i64 add = ((i64)Y0 * (int32_t)(e2 >> 8) + (i64)(((u64)Y0 * (u32)(e2 & 255)) >> 8)) >> 20;
  // 1 / (A 2^-62) = Y 2^-62; a 2^-61 = A 2^-62 2^(1 - y)
  return make_double61(join(Y0, 0) + (u64)add, 63 - y + r);
}

// sqrt(d^2 + c): v = (d^2 + c) / R^2 in units of 2^-63, 2^-10 <= v 2^-63 < 1;
// R = 2^r.
FX_HD double multiquadric(u64 v, int r) {
  const int k = (clz32(hi32(v)) - 1) | 1;
  return make_double61(sqrt60((v << k) >> 4), 62 + (k >> 1) - r);
}

// ------------------------------------------------- scaled 56-bit numbers ---
// Operands of integer products of matrices (digits.cuh): x 2^(56 - e) as an
// integer for |x| <= 2^e, and its seven signed 8-bit digits, the lowest first.
// Of a product x y the digits' products below 256^6 are left out (digits.cuh).
FX_HD u64 abs_bits(double x) { return bits_of(x) & 0x7fffffffffffffffull; }
// e with |x| <= 2^e from the bits of the largest |x|; NOT_FINITE, which makes
// every integer 0 and every scale NaN, if that is infinite or NaN
constexpr int NOT_FINITE = 16384;
FX_HD int scale_exp(u64 maxbits) {
  return maxbits >= 0x7ff0000000000000ull ? NOT_FINITE : (int)(maxbits >> 52) - 1022;
}
// The size of a number is its biased exponent.  Numbers that span ONE_SIZE powers of
// two at most (within a factor of 8) keep FP64's precision in one scale: 56 bits for
// the largest are 53 and more for the smallest.
constexpr int ONE_SIZE = 2;
FX_HD int size_of(double x) { return (int)(abs_bits(x) >> 52); }
FX_HD int size_span(int smallest, int largest) {  // infinite and NaN: no size
  return largest == 2047 ? largest : largest - smallest;
}
FX_HD i64 whole56(double x, int e) {
  const u64 u = bits_of(x);
  const int ex = (int)((u >> 52) & 0x7ff);
  const u64 m = (u & 0xfffffffffffffull) | (ex ? 1ull << 52 : 0ull);
  const int sh = (ex ? ex : 1) - 1075 + 56 - e;  // |x| 2^(56 - e) = m 2^sh, sh <= 4
  i64 f = sh >= 0 ? (i64)(m << sh) : (sh > -63 ? (i64)(((m >> (-sh - 1)) + 1) >> 1) : 0);
  return (u >> 63) ? -f : f;
}
constexpr int DIGITS = 7;
// The digit d of q, d = 0, 1, ... in turn; the last is what is left (at most 256).
FX_HD int next_digit(i64 &q, int d) {
  const int a = d < DIGITS - 1 ? (int)(signed char)(q & 255) : (int)q;
  q = (q - a) >> 8;
  return a;
}
// 2^(e - 56) (2^-1022 at least; infinite from 2^1024 on)
FX_HD double scale56(int e) {
  const int b = e - 56 + 1023;
  if (b > 2046) return from_bits(b > NOT_FINITE / 2 ? 0x7ff8000000000000ull : 0x7ff0000000000000ull);
  return from_bits((u64)(b > 1 ? b : 1) << 52);
}
// 2^k for -1074 <= k <= 1023
FX_HD double pow2(int k) { return from_bits(k >= -1022 ? (u64)(k + 1023) << 52 : 1ull << (k + 1074)); }
// t 2^(e - 56) for a whole number t, rounded once, e the sum of two scales (-2044 at
// least), also where 2^(e - 56) itself is beyond the doubles; NaN if one of the two
// was NOT_FINITE.
FX_HD double times56(double t, int e) {
  const int k = e - 56;
  if (k >= -1022 && k <= 1023) return t * pow2(k);
  if (e > NOT_FINITE / 2) return from_bits(0x7ff8000000000000ull);
  return t * pow2(k / 2) * pow2(k - k / 2);  // the first product is exact, or infinite as the second
}

// ------------------------------------------------------------------- units ---
// The fixed point of one kernel for pairs up to `reach` apart: coordinates
// X = x f 2^k, and the kernel's constant.  ok false: the kernel's
// parameter or the reach is outside what the value functions cover --
//   Gaussian      t = p0 d^2 log2(e) must stay below 1020, where the value is
//                 normal; from 255 on, where 63 bits hold no difference in
//                 units of 2^-59, units of 2^-58 (r = 1);
//   Wendland      q must stay below 1.99 (the same);
//   multiquadric  p0 >= R^2 / 1024: the sum's units show at distance 0 below (at
//                 the limit 2^-52.4 at most and 2^-53.6 rms, as in FP64);
//   Laplace       0 <= p0 < R.
// R = 2^r: the power of two above the reach (above sqrt(reach^2 + p0)).
struct Unit {
  int ok, k, r;
  u64 c;
  Factor f;
};
enum { GAUSSIAN = 1, WENDLAND = 2, LAPLACE = 4, MULTIQUADRIC = 5 };  // as abx.h numbers them

template <int KIND> FX_HD Unit make_unit(double p0, double reach) {
  Unit U;
  U.ok = 0;
  U.k = U.r = 0;
  U.c = 0;
  U.f = make_factor(1.0, 0.0);
  double reach2 = reach * reach;
  if (KIND == MULTIQUADRIC) reach2 += p0;
  if (!(p0 >= 0.0) || !(p0 < 1e200) || !(reach2 > 1e-200) || !(reach2 < 1e200)) return U;
  int e = 0;
  frexp(sqrt(reach2) * (1.0 + 1e-12), &e);
  U.r = e;
  if (KIND == GAUSSIAN) {
    const double most = p0 * reach2 * 1.4426950408889634;
    if (!(p0 > 1e-200) || !(most < 1020.0)) return U;
    // sqrt(p0 log2(e)) as hi + lo: log2(e) as a sum of two doubles, one
    // Newton step on the square root
    const double l = 1.4426950408889634, m = 2.0355273740931033e-17;
    const double ah = p0 * l, al = fma(p0, l, -ah) + p0 * m;
    const double s = sqrt(ah), lo = (fma(-s, s, ah) + al) / (2.0 * s);
    U.f = make_factor(s + lo, lo - ((s + lo) - s));
    U.r = most < 255.0 ? 0 : 1;
    U.k = U.r ? 58 : 59;  // t = sum X^2 in units of 2^-52 or 2^-54
  } else if (KIND == WENDLAND) {
    if (!(p0 > 1e-100) || p0 * p0 * reach2 >= 3.96) return U;
    U.f = make_factor(p0, 0.0);
    U.k = 62;  // q^2 in units of 2^-60
  } else {
    U.k = 62 - e;
    if (KIND == MULTIQUADRIC) {
      if (p0 < ldexp(1.0, 2 * e - 10)) return U;
      U.c = (u64)ldexp(p0, 63 - 2 * e);
    } else if (KIND == LAPLACE) {
      if (p0 >= ldexp(1.0, e)) return U;
      U.c = (u64)to_fixed(p0, U.f, 61 - e);
    } else
      return U;
  }
  U.ok = 1;
  return U;
}
template <int KIND> FX_HD i64 fixed(double x, const Unit &U) { return to_fixed(x, U.f, U.k); }

// What a kernel needs of the unit.
struct Consts {
  u64 c;
  int r;
  double k0;  // value at distance 0 (Laplace)
};
FX_HD Consts consts(const Unit &U, double k0) { return {U.c, U.r, k0}; }

// Points within a unit of each other (2^-62 R) have no difference left.  Laplace:
// from p0 = R / 256 on, 1 / p0 is their value to half an ulp; below, only a point
// with itself has it for sure.
constexpr u64 SAME_PLACE_P0 = 1ull << 53;  // in units of 2^-61 R

// Kernel value of one pair from its differences (diff(); the first dims of
// them).  near: a Laplace pair closer than R / 128 that is left to the FP64 formula on
// the double coordinates, unless it is a point with itself (whose value this is).
template <int KIND>
FX_HD double value(i64 dx, i64 dy, i64 dz, int dims, const Consts &C, const u64 *tab, bool &near) {
  i64 S = 0, T = 0;
  sq_acc(dx, S, T);
  if (dims > 1) sq_acc(dy, S, T);
  if (dims > 2) sq_acc(dz, S, T);
  near = false;
  u64 U = 0;
  if (KIND == LAPLACE || KIND == MULTIQUADRIC) {
    U = sq_low(dx);
    if (dims > 1) U += sq_low(dy);
    if (dims > 2) U += sq_low(dz);
  }
  if (KIND == LAPLACE) {
    near = !laplace_far(S);
    if (near) {  // (looked at in here, not for every pair: 3 %)
      if ((S | T) == 0 && U == 0) near = C.c < SAME_PLACE_P0;
      return C.k0;
    }
    int z;
    const u64 n = norm_d2(S, T, U, z);
    return laplace(n, z, C.c, C.r);
  }
  if (KIND == WENDLAND) return wendland(sq_sum(S, T));
  if (KIND == MULTIQUADRIC) return multiquadric(sq_sum_low<3>(S, T, U) + C.c, C.r);
  if (C.r == 0) return exp2_neg(sq_sum(S, T), tab);
  // wide (make_unit): t = sum X^2 in units of 2^-52
  U = sq_low(dx);
  if (dims > 1) U += sq_low(dy);
  if (dims > 2) U += sq_low(dz);
  return exp2_neg(sq_sum_low<2>(S, T, U), tab);
}

}  // namespace fx
}  // namespace abx
