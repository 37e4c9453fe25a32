"""Searches and sparse products at the edges of their kernels' tiles, units and
sort sizes, against all pairs in FP64."""
import itertools

import numpy as np
import pytest
import torch

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu

# rows, columns (0: the same set), dimension, periodic, clustered, radius
SETS = [(1, 0, 3, False, False, 0.5), (33, 0, 2, True, False, 0.2), (31, 1000, 3, True, False, 0.15),
        (4096, 0, 3, False, False, 0.06), (4097, 0, 2, True, False, 0.02),
        (300, 5000, 3, False, False, 0.3), (2500, 0, 3, True, True, 0.1), (0, 40, 2, False, False, 0.1)]


def _points(n, dim, clustered, rng):
    x = rng.uniform(0, 1, (n, dim))
    if clustered:
        x[: n * 4 // 5] = (0.5 + 0.02 * rng.standard_normal((n * 4 // 5, dim))) % 1.0
    return x


def _pairs(x, y, periodic, r):
    """Per image: squared distances (rows x columns) and which of them count."""
    x, y = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    for shift in itertools.product((-1, 0, 1) if periodic else (0,), repeat=x.shape[1]):
        s = torch.tensor(shift, dtype=torch.float64, device="cuda")
        d2 = torch.zeros(len(x), len(y), dtype=torch.float64, device="cuda")
        for d in range(x.shape[1]):
            d2 += (y[None, :, d] - (x[:, d] + s[d])[:, None]) ** 2
        yield d2, d2 <= r * r


def _set(x, periodic):
    p = ab.Particles(x.shape[1]).set(x)
    return p.init_neighbour_search([0.0] * x.shape[1], [1.0] * x.shape[1], [periodic] * x.shape[1], 10)


@pytest.mark.parametrize("rows,cols,dim,periodic,clustered,r", SETS)
def test_counts_and_lists(rows, cols, dim, periodic, clustered, r):
    rng = np.random.default_rng(rows + cols)
    x = _points(rows, dim, clustered, rng)
    p = _set(_points(cols, dim, clustered, rng) if cols else x, periodic)
    y = p.positions
    want = np.zeros((rows, len(y)), dtype=np.int64)
    for _, near in _pairs(x, y, periodic, r):
        want += near.cpu().numpy()
    assert np.array_equal(ab.radius_count(p, x, r), want.sum(1))
    rowptr, cols_ = ab.radius_query_csr(p, x, r)
    assert rowptr[0] == 0 and np.array_equal(np.diff(rowptr), want.sum(1)) and len(cols_) == rowptr[-1]
    got = np.zeros_like(want)
    np.add.at(got, (np.repeat(np.arange(rows), np.diff(rowptr)), cols_), 1)
    assert np.array_equal(got, want)
    again, same, dx = ab.radius_query_csr(p, x, r, with_dx=True)
    assert np.array_equal(again, rowptr) and np.array_equal(same, cols_)
    assert dx.shape == (len(cols_), dim) and np.all((dx ** 2).sum(1) <= r * r * (1 + 1e-12))


def test_pairs_exactly_at_the_radius():
    """Lattice points: distances are exact, and the pairs at r count."""
    g = np.stack(np.meshgrid(*[np.arange(16) / 16.0] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = _set(g, True)
    inside = sum(a * a + b * b + c * c <= 9 for a, b, c in itertools.product(range(-3, 4), repeat=3))
    assert np.all(ab.radius_count(p, g, 3 / 16) == inside)
    K = ab.create_sparse_operator(p, p, 3 / 16, ab.Kernel.make(ab.K_GAUSSIAN, 1e-9), ab.PREC_FP64)
    assert np.all(np.abs(K * np.ones(len(g)) - inside) < inside * 1e-9)


KINDS = [(ab.K_GAUSSIAN, 3.0), (ab.K_LAPLACE, 0.01), (ab.K_MULTIQUADRIC, 0.05), (ab.K_WENDLAND_C2, None)]


@pytest.mark.parametrize("kind,p0", KINDS)
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("rows,cols,dim,periodic,clustered,r", SETS[:-1])
def test_products(rows, cols, dim, periodic, clustered, r, mixed, kind, p0):
    rng = np.random.default_rng(rows + cols + kind)
    p0 = 1.0 / r if p0 is None else p0
    a = _set(_points(rows, dim, clustered, rng), periodic)
    c = _set(_points(cols, dim, clustered, rng), periodic) if cols else a
    b = rng.standard_normal(cols or rows)
    K = ab.create_sparse_operator(a, c, r, ab.Kernel.make(kind, p0),
                                  ab.PREC_MIXED if mixed else ab.PREC_FP64)
    got = K * b
    bt = torch.from_numpy(b).cuda()
    want, scale, count = 0.0, 0.0, 0.0
    for d2, near in _pairs(a.positions, c.positions, periodic, r):
        if kind == ab.K_GAUSSIAN:
            k = torch.exp(-p0 * d2)
        elif kind == ab.K_LAPLACE:
            k = 1 / (d2.sqrt() + p0)
        elif kind == ab.K_MULTIQUADRIC:
            k = (d2 + p0).sqrt()
        else:
            q = d2.sqrt() * p0
            k = (1 - q).clamp(min=0) ** 4 * (4 * q + 1)
        k = torch.where(near, k, torch.zeros_like(k))
        want = want + k @ bt
        # (a Wendland value near its cut-off is good to the rounding of 1)
        scale = scale + (k + near) @ bt.abs()
        count = count + near.sum(1)
    # a term is good to a few roundings, a sum of n of them to n more; FP32: offsets
    # to 2^-20 of the radius, which 1 / (d + p0) magnifies by up to r / p0 = 30
    unit = 2.0 ** -13 if mixed else (16 + count) * 2.0 ** -52
    err = (torch.from_numpy(got).cuda() - want).abs()
    assert bool((err <= unit * scale).all())


@pytest.mark.parametrize("n", [1, 2, 1024, 1025, 2048, 2049, 4096, 4097, 262144, 262145, 524288, 524289])
@pytest.mark.parametrize("few_cells", [False, True])
def test_cell_order_is_stable(n, few_cells):
    """Storage order: by cell, then by input position, at the sizes where the
    sort changes its launches."""
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 1, (n, 2))
    if few_cells:
        x = (np.floor(x * 3) + 0.37) / 3
    size = max(1, int(np.floor(1.0 / (10.0 / n) ** 0.5)))
    cell = np.floor(x * size).astype(np.int64)
    p = _set(x, False)
    assert np.array_equal(p.ids, np.argsort(cell[:, 0] * size + cell[:, 1], kind="stable"))
