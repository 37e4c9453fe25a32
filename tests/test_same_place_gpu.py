"""Laplace products of points that are closer than the fixed-point coordinates'
unit and yet apart."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu
P0 = 1e-28


@pytest.mark.parametrize("m", [2, 40])
@pytest.mark.parametrize("dim", [1, 3])
@pytest.mark.parametrize("form", ["dense", "sparse", "sparse_self", "fmm"])
def test_near_the_origin(form, dim, m):
    """Rows 1e-27 apart beside a corner of the box; 2 of them are a sparse place,
    40 a whole unit of the sparse product."""
    rng = np.random.default_rng(m)
    x = rng.uniform(0.6, 1.0, (m + 30, dim))
    x[:m] = 0.0
    x[:m, 0] = 1e-27 * rng.permutation(m)
    box = [0.0] * dim, [1.0] * dim, [False] * dim
    p = ab.Particles(dim).set(x)
    kern = ab.Kernel.make(ab.K_LAPLACE, P0)
    if form == "fmm":
        p.init_octree(*box, 200)
        K = ab.create_fmm_operator(p, kern, 3)
    elif form == "dense":
        K = ab.create_dense_operator(p, p, kern)
    else:
        p.init_neighbour_search(*box, 10)
        q = ab.Particles(dim).set(x).init_neighbour_search(*box, 10) if form == "sparse" else p
        K = ab.create_sparse_operator(q, p, 0.3, kern)
    x = p.positions
    d = np.sqrt(((x[:, None, :] - x[None, :, :]) ** 2).sum(2))
    k = 1 / (d + P0)
    if form.startswith("sparse"):
        k = np.where(d <= 0.3, k, 0.0)
    # weights without the corner's first point (its own value, 1e28, would hide the others)
    b = rng.uniform(0.5, 1.0, len(x))
    corner = np.nonzero((x < 1e-20).all(1))[0]
    for i in corner[:4]:
        b[i] = 0.0
        got, want = (K * b)[i], k[i] @ b
        assert abs(got - want) <= 1e-13 * want
        b[i] = 1.0
    assert np.all(np.abs(K * b - k @ b) <= 1e-13 * (k @ b))
