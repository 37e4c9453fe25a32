"""The Schwarz blocks' LU (k_lu_fix) on one block, at the edges of its panels,
column blocks and shared-memory rows: the solution's residual."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 130, 711, 712, 713, 1700])
@pytest.mark.parametrize("kind", [ab.K_GAUSSIAN, ab.K_WENDLAND_C2])
def test_one_block(n, kind):
    rng = np.random.default_rng(n)
    p = ab.Particles(2).set(rng.uniform(0, 1, (n, 2)))
    # the root is always divided: all points in one quadrant make one block
    p.init_octree([0.0, 0.0], [2.0, 2.0], [False, False], 2 * n)
    begin, end = p.tree_leaves()[2:]
    assert np.count_nonzero(end > begin) == 1
    r = 0.4
    p0 = 1.0 / r if kind == ab.K_WENDLAND_C2 else 60.0
    x = p.positions
    d2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(2)
    q = np.minimum(np.sqrt(d2) * p0, 1.0)
    K = np.exp(-p0 * d2) if kind == ab.K_GAUSSIAN else (1 - q) ** 4 * (4 * q + 1)
    K[d2 > r * r] = 0.0
    op = ab.create_sparse_operator(p, p, r, ab.Kernel.make(kind, p0), ab.PREC_FP64)
    b = rng.standard_normal(n)
    y = ab.schwarz_preconditioner(op).solve(b)
    # backward stability with partial pivoting: n roundings of |K| |y| times a
    # growth that stays small for these matrices; and the entries' own rounding,
    # (4 + 2 p0 r^2) 2^-52
    bound = (16 * n + 64) * 2.0 ** -53 * (np.abs(K).sum(1).max() * np.abs(y).max() + np.abs(b).max())
    assert np.abs(K @ y - b).max() <= bound
