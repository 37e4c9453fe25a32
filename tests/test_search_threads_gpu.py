"""Searches of one particle set by several threads, each with host queries of its
own."""
import threading

import numpy as np
import pytest

import aboria_gb300 as ab

pytestmark = pytest.mark.gpu


def test_host_queries_of_several_threads():
    rng = np.random.default_rng(0)
    p = ab.Particles(3).set(rng.uniform(0, 1, (20_000, 3)))
    p.init_neighbour_search([0.0] * 3, [1.0] * 3, [True] * 3, 10)
    queries = [rng.uniform(0, 1, (n, 3)) for n in (1, 700, 3000, 5001)]
    want = [(ab.radius_count(p, q, 0.07), ab.radius_query_csr(p, q, 0.07)) for q in queries]
    wrong = []

    def search(t):
        for k in range(30):
            w = (t + k) % len(queries)
            counts = ab.radius_count(p, queries[w], 0.07)
            rowptr, cols = ab.radius_query_csr(p, queries[w], 0.07)
            if not (np.array_equal(counts, want[w][0]) and np.array_equal(rowptr, want[w][1][0])
                    and np.array_equal(cols, want[w][1][1])):
                wrong.append((t, k))

    threads = [threading.Thread(target=search, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
