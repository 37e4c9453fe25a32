"""What a particle set's searches leave allocated is in proportion to the set."""
import numpy as np
import pytest
import torch

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


def test_many_queries_of_a_small_set():
    rng = np.random.default_rng(0)
    p = ab.Particles(3).set(rng.uniform(0, 1, (1000, 3)))
    p.init_neighbour_search([0.0] * 3, [1.0] * 3, [False] * 3, 10)
    q = torch.rand(8_000_000, 3, dtype=torch.float64, device="cuda")
    counts = torch.empty(len(q), dtype=torch.int32, device="cuda")
    want = ab.radius_count(p, q[:1000].cpu().numpy(), 0.1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        ab.radius_count(p, q, 0.1, out=counts)
        # 8 million queries take about 800 MB while they are searched
        assert torch.cuda.mem_get_info()[0] > before - (64 << 20)
        assert np.array_equal(counts[:1000].cpu().numpy(), want)
