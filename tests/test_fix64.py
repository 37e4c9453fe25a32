"""FP64-accurate kernel values from integer arithmetic (csrc/fix64.cuh), on the
CPU against 50-digit decimals: the same header the GPU kernels include."""
import ctypes as C
import random
import subprocess
from decimal import Decimal, getcontext
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
getcontext().prec = 50
SRC = r"""
#include "fix64.cuh"
using namespace abx::fx;
static constexpr ExpTable TAB = make_exp_table();
template <int KIND> static double run(const double *x, const double *y, int dim, double reach,
                                      double p0) {
  const Unit U = make_unit<KIND>(p0, reach);
  if (!U.ok) return -2.0;
  i64 d[3] = {0, 0, 0};
  for (int k = 0; k < dim; ++k)
    d[k] = diff(fixed<KIND>(y[k], U), biased(fixed<KIND>(x[k], U)));
  bool near;
  const double v = value<KIND>(d[0], d[1], d[2], dim, consts(U, 1.0 / p0), TAB.v, near);
  return near ? -1.0 : v;
}
extern "C" {
double v_gauss(const double *x, const double *y, int dim, double reach, double p0) {
  return run<GAUSSIAN>(x, y, dim, reach, p0);
}
double v_wend(const double *x, const double *y, int dim, double reach, double p0) {
  return run<WENDLAND>(x, y, dim, reach, p0);
}
double v_lap(const double *x, const double *y, int dim, double reach, double p0) {
  return run<LAPLACE>(x, y, dim, reach, p0);
}
// sum of n products of scaled 56-bit numbers
double dot56(const double *x, const double *y, int n) {
  u64 mx = 0, my = 0;
  for (int i = 0; i < n; ++i) {
    mx = abs_bits(x[i]) > mx ? abs_bits(x[i]) : mx;
    my = abs_bits(y[i]) > my ? abs_bits(y[i]) : my;
  }
  const int ex = scale_exp(mx), ey = scale_exp(my);
  i64 w[2 * DIGITS - 1] = {};  // sums by weight
  for (int i = 0; i < n; ++i) {
    i64 a = whole56(x[i], ex), b = whole56(y[i], ey);
    int p[DIGITS], q[DIGITS];
    for (int d = 0; d < DIGITS; ++d) p[d] = next_digit(a, d), q[d] = next_digit(b, d);
    for (int d = 0; d < DIGITS; ++d)
      for (int c = DIGITS - 1 - d; c < DIGITS; ++c) w[c + d] += p[c] * q[d];
  }
  i64 s = w[2 * DIGITS - 2];
  for (int k = 2 * DIGITS - 3; k >= DIGITS; --k) s = s * 256 + w[k];
  s += (w[DIGITS - 1] + 128) >> 8;
  for (int k = DIGITS - 1; k < 2 * DIGITS - 1; ++k)
    if (w[k] > (1 << 24) || -w[k] > (1 << 24)) return 1e300;  // not exact in FP32
  return (double)s * scale56(ex + ey);
}
double v_mq(const double *x, const double *y, int dim, double reach, double p0) {
  return run<MULTIQUADRIC>(x, y, dim, reach, p0);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fix64")
    (d / "fix64_host.cpp").write_text(SRC)
    so = d / "fix64_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    str(ROOT / "aboria_gb300" / "csrc"), str(d / "fix64_host.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    for f in ("v_gauss", "v_wend", "v_lap", "v_mq", "dot56"):
        getattr(lib, f).restype = C.c_double
    return lib


def _exact(kind, x, y, p0):
    d2 = sum((Decimal(b) - Decimal(a)) ** 2 for a, b in zip(x, y))
    p = Decimal(p0)
    if kind == "gauss":
        # beyond p0 d^2 = 177 coordinates are in units of 2^-58: the value's slope,
        # ln 2 2 sqrt(3 t), times a difference's error of up to one unit
        k, t = (-d2 * p).exp(), d2 * p * Decimal("1.443")
        return k, k * t.sqrt() * Decimal(2) ** -55
    if kind == "lap":
        return 1 / (d2.sqrt() + p), Decimal(0)
    if kind == "mq":
        return (d2 + p).sqrt(), Decimal(0)
    q = d2.sqrt() * p
    t = 1 - q
    # the slope of the value times the root's error
    return (t ** 4 * (4 * q + 1), 20 * q * abs(t) ** 3 * Decimal(2) ** -59) if t > 0 else (Decimal(0), Decimal(0))


@pytest.mark.parametrize("kind,p0r2", [("gauss", 4.0), ("gauss", 21.0), ("gauss", 170.0), ("gauss", 180.0), ("gauss", 600.0), ("wend", 1.0),
                                       ("lap", 0.0), ("lap", 1e-11), ("lap", 0.02), ("lap", 0.4),
                                       ("mq", 0.005), ("mq", 0.02), ("mq", 0.7)])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_values_within_an_ulp(lib, kind, p0r2, dim):
    rng = random.Random(7 * dim + len(kind))
    for case in range(300):
        radius = rng.choice([0.02, 0.05, 1.0, 37.0])
        # points of [-4, 4] radii, pairs from nearly touching to the radius
        x = [rng.uniform(-4, 4) * radius for _ in range(dim)]
        dist = radius * 2.0 ** -rng.uniform(0, 9)
        v = [rng.gauss(0, 1) for _ in range(dim)]
        n = sum(c * c for c in v) ** 0.5
        y = [a + dist * 0.999 * c / n for a, c in zip(x, v)]
        p0 = {"gauss": p0r2 / radius ** 2, "wend": p0r2 / radius, "lap": p0r2 * radius,
              "mq": p0r2 * radius ** 2}[kind]
        reach = radius if kind != "mq" else (radius ** 2 + p0) ** 0.5
        r = 0
        while 2.0 ** r < reach * 1.0001:
            r += 1
        while 2.0 ** (r - 1) >= reach * 1.0001:
            r -= 1
        X, Y = (C.c_double * dim)(*x), (C.c_double * dim)(*y)
        got = Decimal(getattr(lib, "v_" + kind)(X, Y, dim, C.c_double(radius), C.c_double(p0)))
        want, slack = _exact(kind, x, y, p0)
        if got == -1:  # left to the FP64 formula: closer than R / 128
            assert kind == "lap" and dist < 2.0 ** (r - 7)
            continue
        assert abs(got - want) <= want * Decimal(2) ** -52 + slack, (case, x, y, p0, got, want)


def test_limits(lib):
    x, far = (C.c_double * 1)(0.25), (C.c_double * 1)(0.25 + 0.5)
    assert lib.v_gauss(x, x, 1, C.c_double(1.0), C.c_double(3.0)) == 1.0
    assert lib.v_wend(x, x, 1, C.c_double(0.5), C.c_double(2.0)) == 1.0
    assert lib.v_wend(x, far, 1, C.c_double(0.5), C.c_double(2.0)) == 0.0     # q = 1
    assert lib.v_mq(x, x, 1, C.c_double(0.5), C.c_double(0.25)) == 0.5
    assert lib.v_lap(x, x, 1, C.c_double(0.5), C.c_double(0.125)) == 8.0


@pytest.mark.parametrize("n", [1, 2, 16, 63, 64])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -300, 2.0 ** 300])
def test_scaled_products(lib, n, scale):
    """n products by digits: each operand good to 2^-57 of the largest, the low
    digits' products (2^-58) left out, one rounding of the sum."""
    rng = random.Random(n)
    for bad in (float("inf"), float("nan")):
        v = lib.dot56((C.c_double * n)(*[bad] * n), (C.c_double * n)(*[1.0] * n), n)
        assert v != v
    assert lib.dot56((C.c_double * n)(*[1e200] * n), (C.c_double * n)(*[1e200] * n), n) == float("inf")
    for _ in range(200):
        x = [rng.choice([-1, 1]) * rng.random() * scale * 2.0 ** -rng.randrange(40) for _ in range(n)]
        y = [rng.choice([-1, 1]) * rng.random() for _ in range(n)]
        got = lib.dot56((C.c_double * n)(*x), (C.c_double * n)(*y), n)
        want = sum(Decimal(a) * Decimal(b) for a, b in zip(x, y))
        big = Decimal(max(map(abs, x))) * Decimal(max(map(abs, y)))
        # (largest within a factor of two of the unit: 2 x 2 for both)
        slack = big * 4 * (n * (Decimal(2) ** -57 * 2 + Decimal(2) ** -58) + Decimal(2) ** -56)
        assert abs(Decimal(got) - want) <= slack + abs(want) * Decimal(2) ** -52
