"""The FP64 M2L by digits, term by term: four boxes in 1-D, whose far pairs go through
one M2L matrix and nothing else but the two interpolations, one source at a time."""
import math

import numpy as np
import pytest

import aboria_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", range(2, 9))
@pytest.mark.parametrize("kind,p0", [(ab.K_LAPLACE, 0.05), (ab.K_MULTIQUADRIC, 0.01)])
def test_single_sources(order, kind, p0):
    rng = np.random.default_rng(order)
    x = (np.arange(4)[:, None] + rng.uniform(0, 1, (4, 8))).reshape(-1, 1) / 4
    p = ab.Particles(1).set(x)
    p.init_octree([0.0], [1.0], [False], 8)
    assert len(p.tree_leaves()[0]) == 4
    K = ab.create_fmm_operator(p, ab.Kernel.make(kind, p0), order)
    box = np.floor(p.positions[:, 0] * 4)
    # sums of |R| over the nodes at either end (Lebesgue constant), and the roundings of
    # two interpolations and one product of `order` terms; operands cut to 40 of their
    # 56 bits would be off by up to 2^-41
    most = 2 / math.pi * math.log(order) + 1
    bound = (8 * order + 32) * most * most * 2.0 ** -53
    assert bound < 2.0 ** -43
    for j in range(32):
        b = np.zeros(32)
        b[j] = rng.uniform(1.0, 2.0)
        got = K * b
        want = oracle.fmm(p.positions, [0.0], [1.0], 8, order, kind, [p0], b)
        far = np.abs(box - box[j]) >= 2
        assert far.sum() in (8, 16)
        assert np.all(np.abs(got - want)[far] <= bound * np.abs(want[far]).max())
