"""Mixed products of the queries that k_pairs_thread walks with a few lanes each
(sets of 50,000 rows and more, where a third of the queries have sparse
surroundings), row by row."""
import numpy as np
import pytest
import torch

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


def _set(x, periodic=False):
    dim = x.shape[1]
    p = ab.Particles(dim).set(x)
    return p.init_neighbour_search([0.0] * dim, [1.0] * dim, [periodic] * dim, 10)


def _kernels(r):
    return [(ab.K_CONST, 0.75), (ab.K_GAUSSIAN, 4.0 / r ** 2), (ab.K_COMPACT_GAUSSIAN, 6.0 / r ** 2),
            (ab.K_LAPLACE, 0.05 * r), (ab.K_MULTIQUADRIC, 0.1 * r * r), (ab.K_WENDLAND_C2, 1.0 / r)]


def _value(kind, p0, d2):
    if kind == ab.K_CONST:
        return torch.full_like(d2, p0)
    if kind in (ab.K_GAUSSIAN, ab.K_COMPACT_GAUSSIAN):
        return torch.exp(-p0 * d2)
    if kind == ab.K_LAPLACE:
        return 1 / (d2.sqrt() + p0)
    if kind == ab.K_MULTIQUADRIC:
        return (d2 + p0).sqrt()
    q = (d2.sqrt() * p0).clamp(max=1.0)
    return (1 - q) ** 4 * (4 * q + 1)


@pytest.mark.parametrize("which", range(6))
def test_sparse_queries_beside_dense_clumps(which):
    """Queries alone in their row of cells, one cell (a radius' third) beside
    clumps of 100,000 columns: all of a row's terms, which are positive, lie in one
    row of its stencil."""
    r, m = 0.04, 74  # cells of side 1 / 74, the 74th part being the first above r / 3
    kind, p0 = _kernels(r)[which]
    rng = np.random.default_rng(1)
    cells = np.array([[15, 15, 15], [55, 15, 50], [15, 55, 55], [55, 55, 30]]) + 0.5
    clumps = (cells[:, None, :] + rng.uniform(-0.1, 0.1, (4, 100_000, 3))) / m
    # three queries (a unit of fewer than four) in each of the four cells beside a
    # clump's, in other rows; and 50,000 with nothing near them
    side = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0]])
    near = ((cells[:, None, :] + side[None])[:, :, None, :] + rng.uniform(-0.1, 0.1, (4, 4, 3, 3))) / m
    far = rng.uniform(0, 1, (60_000, 3))
    far = far[np.abs(far[:, None, :] - cells[None] / m).max(2).min(1) > 2 * r][:50_000]
    rows, cols = _set(np.concatenate([near.reshape(-1, 3), far])), _set(clumps.reshape(-1, 3))
    assert len(rows) == 50_048
    b = rng.uniform(0.5, 1.5, len(cols))
    got = ab.create_sparse_operator(rows, cols, r, ab.Kernel.make(kind, p0), ab.PREC_MIXED) * b
    q = torch.from_numpy(rows.positions).cuda()
    y, bt = torch.from_numpy(cols.positions).cuda(), torch.from_numpy(b).cuda()
    close = ((q[:, None] - torch.from_numpy(cells / m).cuda()[None]).abs().amax(2) < 2 * r).any(1)
    assert int(close.sum()) == 48
    got = torch.from_numpy(got).cuda()
    assert bool((got[~close] == 0).all())
    for i in torch.nonzero(close).flatten():
        d2 = ((y - q[i]) ** 2).sum(1)
        want = (torch.where(d2 <= r * r, _value(kind, p0, d2), 0.0 * d2) * bt).sum()
        # offsets to 6 2^-24 of a cell, at 0.8 cells and more, times a kernel's
        # condition of up to 2.3; a value's 8 roundings; 31 of a block of 32 terms
        assert abs(float(got[i] - want)) <= (17 + 8 + 31) * 2.0 ** -24 * float(want)


@pytest.mark.parametrize("which", range(6))
@pytest.mark.parametrize("dim,n,neighbours,periodic", [(3, 50_000, 9, True), (3, 80_021, 12, False),
                                                      (2, 50_001, 8, True), (3, 330_007, 5, False)])
def test_uniform_sets(which, dim, n, neighbours, periodic):
    """Against the FP64 operator, from the first size that takes this kernel to
    one lane a query."""
    ball = {2: np.pi, 3: 4 / 3 * np.pi}[dim]
    r = (neighbours / n / ball) ** (1 / dim)
    kind, p0 = _kernels(r)[which]
    rng = np.random.default_rng(n)
    p = _set(rng.uniform(0, 1, (n, dim)), periodic)
    b = rng.standard_normal(n)
    kern = ab.Kernel.make(kind, p0)
    got = ab.create_sparse_operator(p, p, r, kern, ab.PREC_MIXED) * b
    exact = ab.create_sparse_operator(p, p, r, kern, ab.PREC_FP64)
    want = exact * b
    ones = ab.create_sparse_operator(p, p, r, ab.Kernel.make(ab.K_CONST, 1.0), ab.PREC_FP64)
    # (a Wendland value near its cut-off is good to the rounding of 1); offsets to
    # 2^-20 of the radius, which 1 / (d + p0) magnifies by up to r / p0 = 20
    assert np.all(np.abs(got - want) <= 2.0 ** -14 * (exact * np.abs(b) + ones * np.abs(b)))
