"""How queries are put into units: sets with one or few columns of cells, and sets
whose sparse queries lie beside dense ones, with kernels that have FP64 values."""
import itertools

import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


def _counts(x, y, length, periodic, r):
    n = np.zeros(len(x), dtype=np.int64)
    for shift in itertools.product((-1, 0, 1) if periodic else (0,), repeat=x.shape[1]):
        for i0 in range(0, len(x), 500):
            d2 = 0.0
            for d, s in enumerate(shift):
                d2 = d2 + (y[None, :, d] - (x[i0:i0 + 500, d] + s * length[d])[:, None]) ** 2
            n[i0:i0 + 500] += (d2 <= r * r).sum(1)
    return n


@pytest.mark.parametrize("own_rows", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("n,length,r", [(1, [1.0], 0.1), (33, [1.0], 0.2), (900, [1.0], 0.003), (4000, [1.0], 0.001),
                                        (4000, [1.0], 0.05), (3000, [1.0, 0.02], 0.01), (3000, [1.0, 0.1], 0.1),
                                        (3000, [1.0, 0.02, 0.02], 0.015)])
def test_few_columns(n, length, r, periodic, own_rows):
    rng = np.random.default_rng(n)
    length = np.array(length)
    x = rng.uniform(0, 1, (n, len(length)))
    x[: n // 3, 0] = 0.4 + 0.01 * x[: n // 3, 0]  # cells of many points too
    q = rng.uniform(0, 1, (n // 2 + 1, len(length))) * length if own_rows else x * length
    box = [0.0] * len(length), length.tolist(), [periodic] * len(length)
    p = ab.Particles(len(length)).set(x * length).init_neighbour_search(*box, 10)
    want = _counts(q, p.positions, length, periodic, r)
    assert np.array_equal(ab.radius_count(p, q, r), want)
    rowptr, cols = ab.radius_query_csr(p, q, r)
    assert np.array_equal(np.diff(rowptr), want) and len(cols) == rowptr[-1]
    rows = ab.Particles(len(length)).set(q).init_neighbour_search(*box, 10) if own_rows else p
    want = _counts(rows.positions, p.positions, length, periodic, r)
    for prec in (ab.PREC_FP64, ab.PREC_MIXED):
        K = ab.create_sparse_operator(rows, p, r, ab.Kernel.make(ab.K_CONST, 1.0), prec)
        assert np.array_equal(K * np.ones(n), want)
    # rows next to one another, as a Wendland sum: one unit's queries and the next's
    kern = ab.Kernel.make(ab.K_WENDLAND_C2, 1.0 / r)
    b = rng.uniform(0.5, 1.0, n)
    got = [ab.create_sparse_operator(rows, p, r, kern, prec) * b for prec in (ab.PREC_FP64, ab.PREC_MIXED)]
    assert np.all(np.abs(got[0] - got[1]) <= 1e-5 * (want + 1))


@pytest.mark.parametrize("dim,n,r", [(2, 6000, 0.02), (3, 6000, 0.08)])
@pytest.mark.parametrize("periodic", [False, True])
def test_sparse_places_beside_dense_ones(dim, n, r, periodic):
    """A constant kernel's FP64 sums of ones are counts, whichever kernel a query goes
    to: alone, beside a cluster (also across the box' edge), or in one."""
    rng = np.random.default_rng(dim)
    x = rng.uniform(0, 1, (n, dim))
    x[: n // 2] = (0.02 * rng.standard_normal((n // 2, dim))) % 1.0
    box = [0.0] * dim, [1.0] * dim, [periodic] * dim
    p = ab.Particles(dim).set(x).init_neighbour_search(*box, 10)
    want = _counts(p.positions, p.positions, np.ones(dim), periodic, r)
    assert np.array_equal(ab.create_sparse_operator(p, p, r, ab.Kernel.make(ab.K_CONST, 1.0)) * np.ones(n), want)
    # the same rows from a set of queries of its own
    q = rng.uniform(0, 1, (900, dim))
    rows = ab.Particles(dim).set(q).init_neighbour_search(*box, 10)
    got = ab.create_sparse_operator(rows, p, r, ab.Kernel.make(ab.K_CONST, 2.0)) * np.ones(n)
    assert np.array_equal(got, 2.0 * _counts(rows.positions, p.positions, np.ones(dim), periodic, r))
