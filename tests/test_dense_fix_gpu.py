"""The dense FP64 product on the integer units (k_dense_fix) against the FP64
formulas in numpy, at the edges of its tiles and of the rule that selects it."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


def _on_integers(x, y, kind, p0):
    """The rule of the kernel's dispatch (R: power of two above the diagonal)."""
    both = np.concatenate([x, y])
    ext2 = ((both.max(0) - both.min(0)) ** 2).sum()
    reach2 = ext2 + (p0 if kind == ab.K_MULTIQUADRIC else 0.0)
    R = 2.0 ** np.ceil(np.log2(np.sqrt(reach2 or 1.0)))
    return {ab.K_GAUSSIAN: p0 * ext2 * 1.4427 < 1020.0, ab.K_LAPLACE: p0 < R,
            ab.K_MULTIQUADRIC: p0 >= R * R / 1024, ab.K_WENDLAND_C2: p0 ** 2 * ext2 < 3.96}[kind]


def _reference(x, y, kind, p0, b):
    # the FP64 formula's argument alone is off by more than the integer path's
    # value: that one is held against extended precision
    real = np.longdouble if _on_integers(x, y, kind, p0) else np.float64
    x, y, b, p0 = x.astype(real), y.astype(real), b.astype(real), real(p0)
    d2 = ((x[:, None, :] - y[None, :, :]) ** 2).sum(2)
    if kind == ab.K_GAUSSIAN:
        k = np.exp(-d2 * p0)
    elif kind == ab.K_LAPLACE:
        with np.errstate(divide="ignore"):
            k = 1.0 / (np.sqrt(d2) + p0)
    elif kind == ab.K_MULTIQUADRIC:
        k = np.sqrt(d2 + p0)
    else:
        q = np.minimum(np.sqrt(d2) * p0, 1.0)
        k = (1 - q) ** 4 * (4 * q + 1)
    with np.errstate(invalid="ignore"):
        return (k * b).sum(1), (np.abs(k) * np.abs(b)).sum(1)


def _run(x, y, kind, p0, b):
    dim = x.shape[1]
    K = ab.create_dense_operator(ab.Particles(dim).set(x), ab.Particles(dim).set(y),
                                 ab.Kernel.make(kind, p0))
    return K * b


# p0 on both sides of the rules: Gaussian p0 diag^2 log2(e) below and above 255 and 1020,
# Wendland support above and below R / 2, softening below and above R
CASES = [(ab.K_GAUSSIAN, 5.0), (ab.K_GAUSSIAN, 400.0), (ab.K_GAUSSIAN, 9000.0),
         (ab.K_LAPLACE, 1e-12), (ab.K_LAPLACE, 0.05), (ab.K_LAPLACE, 9.0), (ab.K_MULTIQUADRIC, 0.1), (ab.K_MULTIQUADRIC, 0.02), (ab.K_MULTIQUADRIC, 1e-4),
         (ab.K_WENDLAND_C2, 0.4), (ab.K_WENDLAND_C2, 3.0)]


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("rows,cols", [(1, 1), (255, 257), (256, 256), (700, 1), (33, 5000)])
@pytest.mark.parametrize("kind,p0", CASES)
def test_matches_fp64_formula(dim, rows, cols, kind, p0):
    rng = np.random.default_rng(100 * dim + rows + cols)
    x, y = rng.uniform(-0.3, 1.2, (rows, dim)), rng.uniform(0, 1, (cols, dim))
    y[: cols // 3] = x[np.arange(cols // 3) % rows]          # coincident points
    y[cols // 3: cols // 2] = x[np.arange(cols // 3, cols // 2) % rows] + 1e-5  # close ones
    b = rng.standard_normal(cols)
    want, scale = _reference(x, y, kind, p0, b)
    # a term is good to a few rounding errors, a sum of n terms to n more
    assert np.all(np.abs(_run(x, y, kind, p0, b) - want) <= (8 + cols) * 2.0 ** -52 * scale)


def test_values_that_are_not_finite_pass_through():
    rng = np.random.default_rng(5)
    x, y, b = rng.uniform(0, 1, (300, 2)), rng.uniform(0, 1, (400, 2)), np.ones(400)
    b[3] = np.inf
    assert np.all(np.isinf(_run(x, y, ab.K_GAUSSIAN, 1.0, b)))
    b[4] = -np.inf
    assert np.all(np.isnan(_run(x, y, ab.K_GAUSSIAN, 1.0, b)))
    b[:] = 1.0
    x[7, 1] = np.nan
    got = _run(x, y, ab.K_MULTIQUADRIC, 1.0, b)
    assert np.isnan(got[7]) and np.isfinite(np.delete(got, 7)).all()
    # coincident points and no softening: the FP64 formula's infinity
    got = _run(y, y, ab.K_LAPLACE, 0.0, b)
    assert np.all(np.isinf(got))
