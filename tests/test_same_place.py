"""Laplace values of points closer than the fixed-point coordinates' unit
(csrc/fix64.cuh), on the CPU: the value at distance 0 only where it is theirs."""
import ctypes as C
import subprocess
from fractions import Fraction
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = r"""
#include "fix64.cuh"
using namespace abx::fx;
static constexpr ExpTable TAB = make_exp_table();
extern "C" double laplace_of(double x, double y, double reach, double p0, int *left_out) {
  const Unit U = make_unit<LAPLACE>(p0, reach);
  bool near;
  const double v = value<LAPLACE>(diff(fixed<LAPLACE>(y, U), biased(fixed<LAPLACE>(x, U))), 0, 0, 1,
                                  consts(U, 1.0 / p0), TAB.v, near);
  *left_out = near;
  return U.ok ? v : -1.0;
}
"""


@pytest.fixture(scope="module")
def laplace(tmp_path_factory):
    d = tmp_path_factory.mktemp("same_place")
    (d / "host.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    str(ROOT / "aboria_gb300" / "csrc"), str(d / "host.cpp"), "-o", str(d / "host.so")],
                   check=True)
    f = C.CDLL(str(d / "host.so")).laplace_of
    f.restype = C.c_double

    def call(x, y, reach, p0):
        out = C.c_int()
        v = f(C.c_double(x), C.c_double(y), C.c_double(reach), C.c_double(p0), C.byref(out))
        return v, bool(out.value)

    return call


@pytest.mark.parametrize("reach", [0.03, 0.9, 50.0])
@pytest.mark.parametrize("p0", [1e-28, 1e-12, 1e-3, 0.004, 0.02, 0.4])
@pytest.mark.parametrize("apart", [1e-27, 1e-21, 1e-20, 3e-20])
def test_points_closer_than_a_unit(laplace, reach, p0, apart):
    p0 *= reach
    v, left_out = laplace(0.0, apart * reach, reach, p0)
    want = 1 / (Fraction(apart * reach) + Fraction(p0))
    assert left_out or abs(Fraction(v) - want) <= want / 2 ** 52
    if left_out:
        assert p0 < reach / 64  # (a larger one hides the distance)


def test_a_point_with_itself(laplace):
    for p0 in (1e-28, 1e-3, 0.4):
        assert laplace(0.3, 0.3, 1.0, p0)[0] == 1.0 / p0
