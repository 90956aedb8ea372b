"""The one-kernel change-tracking pass (one-word tiles of up to 64 - 2k rows)
against the oracle, for every register count it is built for: tiles at the
edges of the grid and of flag words, active runs longer than a window, the
hand-over between dense and tile passes, and chunks of passes in graphs."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


def run(cells, gens, k, tile_rows=0, **kw):
    y, x = cells.shape
    with golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32, temporal_steps=k,
                         algorithm="local", tile_rows=tile_rows, **kw) as e:
        e.set_and_format_input_data(cells)
        e.initialize_data_structures()
        for n in gens:
            e.run(n)
        e.finalize_data_structures()
        return e.fetch_result()


# rows + 2k: 18, 20 (20 in registers); 21, 32 (32); 33, 64 (64); 65 (three kernels)
@pytest.mark.parametrize("k,tile_rows", [(6, 6), (6, 8), (6, 9), (8, 16), (9, 15), (16, 32),
                                         (16, 33), (1, 4), (2, 7)])
@pytest.mark.parametrize("x,y,dense_pct", [(32, 5, 0), (992, 131, 101), (1056, 257, 0),
                                           (2048 + 96, 640, 40)])
def test_vs_oracle(x, y, dense_pct, k, tile_rows):
    rng = np.random.default_rng(x + y + k)
    cells = (rng.random((y, x)) < 0.3).astype(np.uint8)
    cells[y // 3:2 * y // 3, x // 4:] = 0          # a dead part beside an active one
    gens = (23 * k + k // 2, 5 * k)                # graph chunks, single passes, a remainder
    got = run(cells, gens, k, tile_rows, dense_pct=dense_pct)
    assert np.array_equal(got, oracle.life_cells(cells, sum(gens)))


def test_corners_and_word_edges():
    """Blinkers and blocks in the corners and across 32- and 1024-cell edges."""
    y, x = 200, 3200
    cells = np.zeros((y, x), np.uint8)
    for cx in (0, 30, 31, 32, 1022, 1023, 1024, 2047, x - 3):
        for cy in (0, 5, 6, 99, y - 3):
            cells[cy:cy + 3, cx] = 1
    for n in (60, 61, 121):
        assert np.array_equal(run(cells, (n,), 6), oracle.life_cells(cells, n)), n
