"""Dense FP64 products around the size where the one-launch kernel ends, against the
FP64 formula."""
import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu

KERNELS = [(ab.K_GAUSSIAN, 5.0), (ab.K_GAUSSIAN, 4000.0), (ab.K_COMPACT_GAUSSIAN, 30.0), (ab.K_WENDLAND_C2, 1.0),
           (ab.K_WENDLAND_C2, 3.0), (ab.K_LAPLACE, 1e-3), (ab.K_MULTIQUADRIC, 0.01), (ab.K_MULTIQUADRIC, 1e-9)]


@pytest.mark.parametrize("kind,p0", KERNELS)
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("nr,nc", [(1, 1), (1, 2047), (2047, 1), (255, 257), (1024, 1024), (1024, 1025), (300, 1749)])
def test_sizes(nr, nc, dim, kind, p0):
    rng = np.random.default_rng(nr + nc)
    x, y = rng.uniform(0, 1, (nr, dim)), rng.uniform(0, 1, (nc, dim))
    y[: min(nr, nc) // 3] = x[: min(nr, nc) // 3]
    b = rng.standard_normal(nc)
    K = ab.create_dense_operator(ab.Particles(dim).set(x), ab.Particles(dim).set(y), ab.Kernel.make(kind, p0))
    d2 = ((x[:, None, :] - y[None, :, :]) ** 2).sum(2)
    q = np.minimum(np.sqrt(d2) * p0, 1.0)
    k = {ab.K_GAUSSIAN: np.exp(-p0 * d2), ab.K_COMPACT_GAUSSIAN: np.exp(-p0 * d2),
         ab.K_WENDLAND_C2: (1 - q) ** 4 * (4 * q + 1), ab.K_LAPLACE: 1 / (np.sqrt(d2) + p0),
         ab.K_MULTIQUADRIC: np.sqrt(d2 + p0)}[kind]
    # a value's roundings (a Gaussian's exponent to 3 2^-53 of itself; Wendland's t to
    # 2^-52) and those of a sum of nc terms
    slack = 3 * p0 * d2 * k if kind in (ab.K_GAUSSIAN, ab.K_COMPACT_GAUSSIAN) else 0.0
    slack = 40 * (1 - q) ** 3 if kind == ab.K_WENDLAND_C2 else slack
    bound = ((16 + nc) * k + slack) @ np.abs(b) * 2.0 ** -52
    assert np.all(np.abs(K * b - k @ b) <= bound)
    # a coordinate that is not a number: its row alone
    x[nr // 2, dim - 1] = np.nan
    got = ab.create_dense_operator(ab.Particles(dim).set(x), ab.Particles(dim).set(y), ab.Kernel.make(kind, p0)) * b
    keep = np.arange(nr) != nr // 2
    assert np.all(np.abs(got - k @ b)[keep] <= bound[keep])
    # (Wendland's q >= 1 is false for it)
    assert np.isnan(got[nr // 2])
