"""Threads that fetch the grids of one batch at the same time get their own
grid's cells, whatever its size beside the others'."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 8])
def test_concurrent_fetches(threads):
    # ascending sizes: later grids are larger than any fetched before
    jobs = [(oracle.random_ones_zeros(32 * (1 + 7 * i), 40 + 90 * i, i), 5 + i) for i in range(16)]
    want = [oracle.life_cells(c, n) for c, n in jobs]
    with golb200.GolBatch() as b:
        ids = [b.add(c, n) for c, n in jobs]
        b.run()
        b.sync()

        def fetch_all(first):
            order = [(first + j) % len(ids) for j in range(len(ids))]
            return all(np.array_equal(b.fetch(ids[i]), want[i]) for _ in range(10) for i in order)

        with ThreadPoolExecutor(max_workers=threads) as pool:
            assert all(pool.map(fetch_all, range(threads)))
