"""Wendland values of very close pairs from integer arithmetic (csrc/fix64.cuh), on
the CPU."""
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
extern "C" {
double wendland_of_square(u64 q2) { return wendland(q2); }
double wendland_of(double x, double y, double reach, double p0) {
  const Unit U = make_unit<WENDLAND>(p0, reach);
  bool near;
  return value<WENDLAND>(diff(fixed<WENDLAND>(y, U), biased(fixed<WENDLAND>(x, U))), 0, 0, 1,
                         consts(U, 0.0), nullptr, near);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("close")
    (d / "host.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    str(ROOT / "aboria_gb300" / "csrc"), str(d / "host.cpp"), "-o", str(d / "host.so")],
                   check=True)
    lib = C.CDLL(str(d / "host.so"))
    lib.wendland_of.restype = C.c_double
    lib.wendland_of_square.restype = C.c_double
    return lib


def test_squares(lib):
    """Every power of two, its neighbours, and all small numbers, as q^2 2^60."""
    rng = random.Random(0)
    cases = list(range(300)) + [2 ** b + o for b in range(2, 60) for o in (-1, 0, 1)]
    cases += [rng.randrange(2 ** b, 2 ** (b + 1)) for b in range(60) for _ in range(50)]
    for u in cases:
        q = (Decimal(u) / 2 ** 60).sqrt()
        want = (1 - q) ** 4 * (4 * q + 1)
        got = Decimal(lib.wendland_of_square(C.c_uint64(u)))
        assert abs(got - want) <= want * Decimal(2) ** -52 + 20 * q * (1 - q) ** 3 * Decimal(2) ** -59, u


@pytest.mark.parametrize("power", range(-40, 0))
def test_values(lib, power):
    rng = random.Random(power)
    for _ in range(50):
        r = rng.choice([0.05, 1.0, 3e4])
        x = rng.uniform(0, 1) * r
        y = x + r * 2.0 ** power * rng.uniform(0.5, 0.99)
        q = (Decimal(y) - Decimal(x)) * Decimal(1.0 / r)
        want = (1 - q) ** 4 * (4 * q + 1)
        got = Decimal(lib.wendland_of(C.c_double(x), C.c_double(y), C.c_double(r), C.c_double(1.0 / r)))
        assert abs(got - want) <= want * Decimal(2) ** -52 + 20 * q * (1 - q) ** 3 * Decimal(2) ** -59
