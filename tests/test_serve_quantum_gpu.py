"""A quantum below the deepest pass: a round advances no more than it."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quantum,rounds", [(4, 16), (5, 16), (7, 16), (8, 8), (15, 8), (16, 4), (64, 1)])
def test_rounds_of_a_request(quantum, rounds):
    cells = oracle.random_ones_zeros(320, 200, quantum)
    with golb200.GolServer(arena_bytes=1 << 20, quantum=quantum) as s:
        i = s.submit(cells, 64)
        done = []
        while not done:
            s.step()
            done = s.finished()
        assert s.stats()["rounds"] == rounds
        assert np.array_equal(s.fetch(i), oracle.life_cells(cells, 64))
