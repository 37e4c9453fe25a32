"""FP64 FMM products whose M2L matrices hold values of many sizes (k_m2l64), alone
and beside matrices that go by digits."""
import numpy as np
import pytest

import aboria_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p0", [3.0, 300.0])
@pytest.mark.parametrize("dim,order", [(1, 2), (1, 8), (2, 3), (2, 5), (2, 8), (3, 2), (3, 3), (3, 5)])
def test_broad_gaussians(dim, order, p0):
    """p0 = 3: wide matrices on the coarse levels, rows of one size on the fine
    ones; 300: wide ones nearly everywhere, with entries that underflow."""
    n = 3000 if dim < 3 else 1500
    rng = np.random.default_rng(dim * 10 + order)
    p = ab.Particles(dim).set(rng.uniform(0, 1, (n, dim)))
    p.init_octree([0.0] * dim, [1.0] * dim, [False] * dim, 20)
    b = rng.uniform(0.1, 1.0, n)
    got = ab.create_fmm_operator(p, ab.Kernel.make(ab.K_GAUSSIAN, p0), order) * b
    want = oracle.fmm(p.positions, [0.0] * dim, [1.0] * dim, 20, order, ab.K_GAUSSIAN, [p0], b)
    # as for the products by digits: two sums of at most 216 terms, 189 pairs and
    # 1,500 sources a target, and interpolations that may be 50 times the result
    assert np.linalg.norm(got - want) <= 50 * 2000 * 2.0 ** -53 * np.linalg.norm(want)


@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("kind,p0", [(ab.K_LAPLACE, 0.1), (ab.K_GAUSSIAN, 40.0)])
@pytest.mark.parametrize("power", [-1000, -960, 960])
def test_tiny_and_huge_weights(order, kind, p0, power):
    """A power of two on the weights is one on the product, as long as that is
    normal: also where the scale of an M2L product is below 2^-1022."""
    rng = np.random.default_rng(order)
    p = ab.Particles(3).set(rng.uniform(0, 1, (3000, 3)))
    p.init_octree([0.0] * 3, [1.0] * 3, [False] * 3, 20)
    b = rng.uniform(0.5, 1.0, 3000)
    K = ab.create_fmm_operator(p, ab.Kernel.make(kind, p0), order)
    want = K * b
    # only the order of the pairs' sums differs from run to run
    assert np.all(np.abs((K * (b * 2.0 ** power)) * 2.0 ** -power - want) <= 1e-12 * want)
