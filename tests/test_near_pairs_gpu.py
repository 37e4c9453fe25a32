"""FP64 Laplace products of clumps that are small against the radius, so that many
or all of a row's pairs are too close for the fixed-point values."""
import itertools

import numpy as np
import pytest
import torch

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p0", [1e-9, 1e-3])
@pytest.mark.parametrize("own_rows", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dim,clump,size", [(1, 100, 1e-3), (2, 300, 1e-4), (2, 300, 3e-3), (3, 5, 1e-4),
                                            (3, 200, 2e-3), (3, 200, 5e-3)])
def test_clumps(dim, clump, size, periodic, own_rows, p0):
    """Radius 0.1: pairs closer than 1 / 1024 go by FP64.  Clumps of 5 are sparse
    places (a few lanes a query); one clump lies across the box' corner."""
    r, rng = 0.1, np.random.default_rng(clump)
    centres = np.concatenate([np.zeros((1, dim)), rng.uniform(0, 1, (9, dim))])
    x = (centres[:, None, :] + size * rng.uniform(-0.5, 0.5, (10, clump, dim))).reshape(-1, dim) % 1.0
    box = [0.0] * dim, [1.0] * dim, [periodic] * dim
    cols = ab.Particles(dim).set(x).init_neighbour_search(*box, 10)
    rows = cols
    if own_rows:
        rows = ab.Particles(dim).set(x[: len(x) // 2]).init_neighbour_search(*box, 10)
    b = rng.standard_normal(len(cols))
    got = ab.create_sparse_operator(rows, cols, r, ab.Kernel.make(ab.K_LAPLACE, p0)) * b
    q, y = torch.from_numpy(rows.positions).cuda(), torch.from_numpy(cols.positions).cuda()
    bt = torch.from_numpy(b).cuda()
    want = scale = count = 0.0
    for shift in itertools.product((-1, 0, 1) if periodic else (0,), repeat=dim):
        d2 = torch.zeros(len(q), len(y), dtype=torch.float64, device="cuda")
        for d in range(dim):
            d2 += (y[None, :, d] - (q[:, d] + float(shift[d]))[:, None]) ** 2
        near = d2 <= r * r
        k = torch.where(near, 1 / (d2.sqrt() + p0), 0.0 * d2)
        # a shifted coordinate is good to 2^-53 of the box, 2 of them a distance
        off = torch.where(near, 4 * dim * 2.0 ** -53 * k * k, 0.0 * d2) if any(shift) else 0.0
        want, scale = want + k @ bt, scale + (k + 2.0 ** 52 / 16 * off) @ bt.abs()
        count = count + near.sum(1)
    err = (torch.from_numpy(got).cuda() - want).abs()
    assert bool((err <= (16 + count) * 2.0 ** -52 * scale).all())
