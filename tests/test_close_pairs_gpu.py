"""FP64 products of pairs that are very close, far below their distances to others."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,p0", [(ab.K_WENDLAND_C2, 1.0), (ab.K_GAUSSIAN, 4.0), (ab.K_LAPLACE, 0.01), (ab.K_MULTIQUADRIC, 0.1)])
@pytest.mark.parametrize("dim,per_place", [(1, 2), (2, 2), (3, 2), (3, 40)])
@pytest.mark.parametrize("form", ["sparse", "dense"])
def test_pairs_from_one_unit_to_the_radius(form, dim, per_place, kind, p0):
    """Places of 2 points (or 40, a whole unit of the sparse product) at distances of
    2^-45 to 2^-2 of the radius."""
    r, rng = 0.05, np.random.default_rng(dim)
    p0 = {ab.K_WENDLAND_C2: p0 / r, ab.K_LAPLACE: p0 * r}.get(kind, p0 / r ** 2 if kind == ab.K_GAUSSIAN else p0 * r * r)
    size = r * 2.0 ** -np.repeat(np.arange(2, 46), 3)
    x = rng.uniform(0.1, 0.9, (len(size), 1, dim))
    step = rng.standard_normal((len(size), per_place, dim))
    x = (x + size[:, None, None] * step / np.abs(step).max() * (np.arange(per_place) > 0)[None, :, None]).reshape(-1, dim)
    p = ab.Particles(dim).set(x)
    kern = ab.Kernel.make(kind, p0)
    if form == "sparse":
        p.init_neighbour_search([0.0] * dim, [1.0] * dim, [False] * dim, 10)
        K = ab.create_sparse_operator(p, p, r, kern)
    else:
        K = ab.create_dense_operator(p, p, kern)
    x = p.positions
    d2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(2)
    q = np.minimum(np.sqrt(d2) * p0, 1.0)
    k = {ab.K_GAUSSIAN: np.exp(-p0 * d2), ab.K_WENDLAND_C2: (1 - q) ** 4 * (4 * q + 1),
         ab.K_LAPLACE: 1 / (np.sqrt(d2) + p0), ab.K_MULTIQUADRIC: np.sqrt(d2 + p0)}[kind]
    near = d2 <= r * r if form == "sparse" else np.ones_like(d2, dtype=bool)
    k = np.where(near, k, 0.0)
    b = rng.uniform(0.5, 1.0, len(x))
    # roundings of a value (a Gaussian's exponent to 3 2^-53 of itself, Wendland's t to
    # 2^-52 of 1) and of a row's sum
    slack = (3 * p0 * d2 * k if kind == ab.K_GAUSSIAN else 40 * (1 - q) ** 3 * near if kind == ab.K_WENDLAND_C2 else 0 * d2)
    bound = ((16 + near.sum(1))[:, None] * k + slack) @ b * 2.0 ** -52
    assert np.all(np.abs(K * b - k @ b) <= bound)
