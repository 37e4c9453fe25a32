"""FMM products at the edges of their kernels: a near field alone against the
direct sum, and weights far from 1 through the scaled FP16 M2L."""
import numpy as np
import pytest

import aboria_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(1, 1), (1, 70), (2, 33), (2, 150), (3, 64), (3, 400)])
@pytest.mark.parametrize("kind,p0", [(ab.K_LAPLACE, 0.01), (ab.K_MULTIQUADRIC, 0.05), (ab.K_GAUSSIAN, 2.0)])
def test_near_field_alone_is_the_direct_sum(dim, n, kind, p0):
    rng = np.random.default_rng(n)
    # two boxes a dimension: every leaf touches every other one
    p = ab.Particles(dim).set(rng.uniform(0, 1, (n, dim)))
    p.init_octree([0.0] * dim, [1.0] * dim, [False] * dim, n)
    b = rng.standard_normal(n)
    got = ab.create_fmm_operator(p, ab.Kernel.make(kind, p0), 3, ab.PREC_FP64) * b
    x = p.positions
    d2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(2)
    k = {ab.K_LAPLACE: 1 / (np.sqrt(d2) + p0), ab.K_MULTIQUADRIC: np.sqrt(d2 + p0),
         ab.K_GAUSSIAN: np.exp(-p0 * d2)}[kind]
    assert np.all(np.abs(got - k @ b) <= (16 + n) * 2.0 ** -52 * (k @ np.abs(b)))


@pytest.mark.parametrize("order", [5, 6, 7, 8])
def test_mixed_product_of_scaled_weights(order):
    """Powers of two scale the result; weights that span 2^60 over the box keep
    the mixed product within 1e-5 of the FP64 one."""
    rng = np.random.default_rng(order)
    p = ab.Particles(3).set(rng.uniform(0, 1, (6000, 3)))
    p.init_octree([0.0] * 3, [1.0] * 3, [False] * 3, 32)
    kern = ab.Kernel.make(ab.K_LAPLACE, 0.1)
    mixed = ab.create_fmm_operator(p, kern, order, ab.PREC_MIXED)
    exact = ab.create_fmm_operator(p, kern, order, ab.PREC_FP64)
    b = rng.standard_normal(6000)
    for w in (b, b * 2.0 ** 60, b * 2.0 ** -60, b * 2.0 ** (60 * (p.positions[:, 0] - 0.5)), 0 * b):
        want = exact * w
        assert np.linalg.norm(mixed * w - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("dim,order", [(1, 8), (2, 5), (2, 6), (2, 8), (3, 3), (3, 4), (3, 6)])
def test_fp64_m2l_by_digits(dim, order):
    """Node counts around the M2L kernel's 16, 32, 64 and 128 terms (8, 25, 36, 64,
    27, 64, 216), tiles that are not full, weights over many magnitudes."""
    n = 3000 if dim < 3 else 1500
    rng = np.random.default_rng(dim * 10 + order)
    x = rng.uniform(0, 1, (n, dim))
    p = ab.Particles(dim).set(x)
    p.init_octree([0.0] * dim, [1.0] * dim, [False] * dim, 20)
    b = rng.standard_normal(n) * 2.0 ** rng.integers(-20, 1, n)
    got = ab.create_fmm_operator(p, ab.Kernel.make(ab.K_MULTIQUADRIC, 0.01), order) * b
    want = oracle.fmm(p.positions, [0.0] * dim, [1.0] * dim, 20, order, ab.K_MULTIQUADRIC, [0.01], b)
    # two sums of at most 216 terms, 189 pairs and 1,500 sources a target, with up to
    # 50 times the result's size in the terms of signed weights
    assert np.linalg.norm(got - want) <= 50 * 2000 * 2.0 ** -53 * np.linalg.norm(want)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("order", [3, 5])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_weights_that_are_not_finite_reach_every_target(order, mixed, value):
    rng = np.random.default_rng(order)
    p = ab.Particles(3).set(rng.uniform(0, 1, (2000, 3)))
    p.init_octree([0.0] * 3, [1.0] * 3, [False] * 3, 20)
    b = rng.uniform(1, 2, 2000)
    K = ab.create_fmm_operator(p, ab.Kernel.make(ab.K_MULTIQUADRIC, 0.01), order,
                               ab.PREC_MIXED if mixed else ab.PREC_FP64)
    assert np.all(np.isfinite(K * b))
    b[7] = value
    assert not np.any(np.isfinite(K * b))
