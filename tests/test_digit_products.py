"""Products by digits (csrc/fix64.cuh, csrc/digits.cuh) on the CPU: against FP64
sums for rows of numbers of one size, which is what the FMM gives them, and at
the digits' extremes."""
import ctypes as C
import math
import random
import subprocess
from fractions import Fraction
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = r"""
#include "fix64.cuh"
using namespace abx::fx;
extern "C" {
int span(const double *x, int n) {
  int lo = 2047, hi = 0;
  for (int i = 0; i < n; ++i) {
    const int e = size_of(x[i]);
    lo = e < lo ? e : lo;
    hi = e > hi ? e : hi;
  }
  return size_span(lo, hi);
}
int one_size() { return ONE_SIZE; }
// sum of n products of scaled 56-bit numbers, as k_m2l_fix forms it
double dot56(const double *x, const double *y, int n) {
  u64 mx = 0, my = 0;
  for (int i = 0; i < n; ++i) {
    mx = abs_bits(x[i]) > mx ? abs_bits(x[i]) : mx;
    my = abs_bits(y[i]) > my ? abs_bits(y[i]) : my;
  }
  const int ex = scale_exp(mx), ey = scale_exp(my);
  i64 w[2 * DIGITS - 1] = {};
  for (int i = 0; i < n; ++i) {
    i64 a = whole56(x[i], ex), b = whole56(y[i], ey);
    int p[DIGITS], q[DIGITS];
    for (int d = 0; d < DIGITS; ++d) p[d] = next_digit(a, d), q[d] = next_digit(b, d);
    for (int d = 0; d < DIGITS; ++d)
      for (int c = DIGITS - 1 - d; c < DIGITS; ++c) w[c + d] += p[c] * q[d];
  }
  i64 s = w[2 * DIGITS - 2];
  for (int k = 2 * DIGITS - 3; k >= DIGITS; --k) s = s * 256 + w[k];
  return (double)(s + ((w[DIGITS - 1] + 128) >> 8)) * scale56(ex + ey);
}
double scaled(double t, int e) { return times56(t, e); }
double dot64(const double *x, const double *y, int n) {
  double s = 0;
  for (int i = 0; i < n; ++i) s = __builtin_fma(x[i], y[i], s);
  return s;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("digits")
    (d / "digits_host.cpp").write_text(SRC)
    so = d / "digits_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    str(ROOT / "aboria_gb300" / "csrc"), str(d / "digits_host.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.dot56.restype = lib.dot64.restype = lib.scaled.restype = C.c_double
    return lib


def _errors(lib, x, y):
    n = len(x)
    X, Y = (C.c_double * n)(*x), (C.c_double * n)(*y)
    want = sum((Fraction(a) * Fraction(b) for a, b in zip(x, y)), Fraction(0))
    size = sum((abs(Fraction(a) * Fraction(b)) for a, b in zip(x, y)), Fraction(0))
    return [float(abs(Fraction(f(X, Y, n)) - want) / size) for f in (lib.dot56, lib.dot64)], lib.span(X, n)


def _row(kind, n, rng):
    """Kernel values between a target and n points of a box one to two boxes away,
    or any numbers of one size."""
    if kind == "random":
        e = rng.randrange(-200, 200)
        return [math.ldexp(rng.choice([-1, 1]) * rng.uniform(1.0, 2.0), e + rng.randrange(3)) for _ in range(n)]
    d2 = [(1 + rng.random()) ** 2 + rng.uniform(-1, 1) ** 2 + rng.uniform(-1, 1) ** 2 for _ in range(n)]
    if kind == "laplace":
        return [1 / (math.sqrt(v) + 1e-3) for v in d2]
    return [math.sqrt(v + 0.01) for v in d2] if kind == "multiquadric" else [math.exp(-20 * v) for v in d2]


@pytest.mark.parametrize("n", [9, 27, 64, 125])
@pytest.mark.parametrize("weights", ["signed", "positive", "graded"])
@pytest.mark.parametrize("kind", ["laplace", "multiquadric", "random", "gaussian"])
def test_no_further_off_than_fp64(lib, kind, weights, n):
    """Root mean square error relative to the terms' sizes: by digits no larger than
    an FP64 sum's where the rule sends the row to the digits; rows that it keeps
    from them are further off (what the rule is for)."""
    rng = random.Random(n)
    digits = fp64 = 0.0
    for _ in range(400):
        x = _row(kind, n, rng)
        y = [rng.gauss(0, 1) for _ in range(n)]
        if weights == "positive":
            y = [abs(v) for v in y]
        if weights == "graded":  # small where the row is large
            top = max(map(abs, x))
            y = [v * top / abs(k) for v, k in zip(y, x)]
        (a, b), span = _errors(lib, x, y)
        assert (span <= lib.one_size()) == (kind != "gaussian")
        digits += a * a
        fp64 += b * b
    if kind != "gaussian":
        assert digits <= fp64
    elif weights == "graded":
        assert digits > 100 * fp64


def test_sizes(lib):
    inf, nan = float("inf"), float("nan")
    for row, span in (([0.0] * 3, 0), ([1.0, -1.9, 1.5], 0), ([1.0, 7.9], 2), ([1.0, 8.0], 3),
                      ([0.0, 1.0], 1023), ([inf] * 2, 2047), ([nan, 1.0], 2047)):
        assert lib.span((C.c_double * len(row))(*row), len(row)) == span


def _with_digits(d):
    """The number below 1 whose 56-bit integer has these digits, lowest first."""
    return math.ldexp(float(sum(v << (8 * k) for k, v in enumerate(d))), -56)


@pytest.mark.parametrize("digits", [[120, 127, 127, 127, 127, 127, 255], [0, -128, -128, -128, -128, -128, 256],
                                    [8, 127, 127, 127, 127, 127, 128]])
@pytest.mark.parametrize("n", [1, 64, 128])
def test_extreme_digits(lib, digits, n):
    """Largest digits in every place: 128 terms of the weights above the lowest stay
    within 2^24, and what is left out of a term is below 2^-55 of its full scale."""
    x = _with_digits(digits)
    d = list(digits)
    for w in range(7, 13):
        assert n * abs(sum(d[i] * d[w - i] for i in range(7) if 0 <= w - i < 7)) <= 2 ** 24
    got = lib.dot56((C.c_double * n)(*[x] * n), (C.c_double * n)(*[x] * n), n)
    want = n * Fraction(x) ** 2
    assert abs(Fraction(got) - want) <= n * Fraction(1, 2 ** 55) + want / 2 ** 53


@pytest.mark.parametrize("e", [-2044, -1500, -1140, -1100, -1074, -966, -965, 0, 1079, 1080, 1500, 2000])
def test_scales_beyond_the_doubles(lib, e):
    for t in (0, 1, 3, 2 ** 53 - 1, -(2 ** 62), 2 ** 66):
        got = lib.scaled(C.c_double(float(t)), e)
        want = Fraction(t) * Fraction(2) ** (e - 56)
        if abs(want) >= Fraction(2) ** 1024:
            assert got == math.copysign(float("inf"), t)
        else:
            assert got == float(want)  # (Fraction rounds once)
    assert math.isnan(lib.scaled(C.c_double(1.0), 16384 + 5))
