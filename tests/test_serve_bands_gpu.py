"""Served requests whose items' bands follow the load: few items where many
requests run, and the same cells whatever bands a request's rounds had, with
change flags that a change of bands makes stale."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


def serve_all(s, ids, want):
    left = set(ids)
    while left:
        s.step()
        for i in s.finished():
            assert np.array_equal(s.fetch(i), want[i]), i
            left.remove(i)


def test_many_requests_take_tall_bands():
    n, x, y, gens = 48, 1024, 1024, 64
    cells = oracle.random_ones_zeros(x, y, 3)
    end = oracle.life_cells(cells, gens)
    with golb200.GolServer(arena_bytes=256 << 20, quantum=64) as s:
        s.set_tracking("off")
        ids = [s.submit(cells, gens) for _ in range(n)]
        serve_all(s, ids, {i: end for i in ids})
        computed = s.tiles()["computed"]
    tallest = n * (gens // 8) * -(-y // 48) * 2   # bands of 48 rows, two slices of 16 words
    assert tallest <= computed <= 2 * tallest     # 24 rows at least (8-row ones: 5.8 times)


def settling(x, y, seed):
    """Dead but for blinkers, blocks and one region that stays lively for long."""
    cells = np.zeros((y, x), np.uint8)
    r = np.random.RandomState(seed)
    for _ in range(12):
        j, i = r.randint(2, y - 3), r.randint(2, x - 3)
        cells[j, i - 1:i + 2] = 1
    cells[y // 2:y // 2 + 24, x // 2:x // 2 + 40] = oracle.random_ones_zeros(64, 24, seed)[:, :40]
    return cells


@pytest.mark.parametrize("mode", ["on", "auto", "off"])
def test_bands_change_while_a_request_runs(mode):
    shapes = [(1600, 700, 643), (608, 333, 400), (2048, 257, 512), (96, 90, 636)]
    with golb200.GolServer(arena_bytes=256 << 20, quantum=16) as s:
        s.set_tracking(mode)
        want, ids = {}, []

        def submit(cells, gens, end):
            i = s.submit(cells, gens)
            want[i] = end
            ids.append(i)

        for j, (x, y, gens) in enumerate(shapes):
            cells = settling(x, y, j)
            submit(cells, gens, oracle.life_cells(cells, gens))
        done = {}

        def rounds(n):
            for _ in range(n):
                s.step()
                for i in s.finished():
                    done[i] = s.fetch(i)

        load = oracle.random_ones_zeros(2048, 1024, 9)
        load_end = oracle.life_cells(load, 32)
        for burst in range(3):       # alone, beside large requests, alone again
            rounds(5)
            for _ in range(24):
                submit(load, 32, load_end)
            rounds(5)
        while len(done) < len(ids):
            rounds(1)
        for i in ids:
            assert np.array_equal(done[i], want[i]), i
