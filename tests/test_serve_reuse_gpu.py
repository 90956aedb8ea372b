"""A slot freed by a request that was found still, taken by another while the
rounds queued for the first are still running: the newcomer's cells stay its
own (it reaches over the place of the first one's flags)."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


def test_slot_of_a_still_request():
    slow = oracle.random_ones_zeros(4096, 4096, 1)
    still = np.zeros((256, 512), np.uint8)
    still[100:102, 200:202] = 1                       # a block
    newcomer = oracle.random_ones_zeros(640, 512, 2)
    want = oracle.life_cells(newcomer, 8)
    with golb200.GolServer(arena_bytes=64 << 20, quantum=1024) as s:
        s.set_tracking("on")
        s.submit(slow, 8 * 1024)                      # (its rounds take milliseconds)
        first = s.submit(still, 8 * 1024)
        for _ in range(3):
            s.step()
        done = []
        while first not in done:
            done += s.finished()
        assert np.array_equal(s.fetch(first), still)
        assert s.tiles()["early_finished"] == 1
        second = s.submit(newcomer, 8)
        done = []
        while second not in done:
            s.step()
            done += s.finished()
        assert np.array_equal(s.fetch(second), want)
