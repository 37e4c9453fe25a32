"""Mixed products of a Wendland kernel whose support 1 / p0 is wider than the
search radius: its value jumps to 0 at the cut-off."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p0r", [0.3, 0.8, 0.999, 1.0, 1.7])
@pytest.mark.parametrize("dim,n,neighbours,periodic,clustered",
                         [(3, 3000, 40, True, False), (2, 3001, 30, False, True), (3, 50_001, 9, True, False),
                          (2, 60_000, 8, False, False), (3, 60_000, 10, True, True)])
def test_cut_off_inside_the_support(dim, n, neighbours, periodic, clustered, p0r):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 1, (n, dim))
    if clustered:
        x[: n // 2] = (0.5 + 0.05 * rng.standard_normal((n // 2, dim))) % 1.0
    r = (neighbours / n / {2: np.pi, 3: 4 / 3 * np.pi}[dim]) ** (1 / dim)
    p = ab.Particles(dim).set(x)
    p.init_neighbour_search([0.0] * dim, [1.0] * dim, [periodic] * dim, 10)
    b = rng.standard_normal(len(p))
    kern = ab.Kernel.make(ab.K_WENDLAND_C2, p0r / r)
    got = ab.create_sparse_operator(p, p, r, kern, ab.PREC_MIXED) * b
    exact = ab.create_sparse_operator(p, p, r, kern, ab.PREC_FP64)
    ones = ab.create_sparse_operator(p, p, r, ab.Kernel.make(ab.K_CONST, 1.0), ab.PREC_FP64)
    # offsets to 2^-20 of the radius, times a slope of up to 2.1 p0; a value's 8
    # roundings and 31 of a block: near the end of the support all of it absolute
    unit = 2.1 * 1.7 * 2.0 ** -20 + 40 * 2.0 ** -24
    assert np.all(np.abs(got - exact * b) <= 2 * unit * (ones * np.abs(b)))
