"""Depth-4 passes and runs on grids large enough for the row-pair pipeline:
rows as they are (one pass) and interleaved (runs of more than 32 passes),
x-slices, ragged last bands, lanes that do not fill warps and remainders."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu

SHAPES = [(16384, 16384), (16384, 16001), (16000, 17003), (32768, 16386), (33280, 15000)]


@pytest.mark.parametrize("x,y", SHAPES)
def test_pass_vs_oracle(x, y):
    import torch
    rows = np.random.default_rng(x + y).integers(0, 1 << 32, (y, x // 32), dtype=np.uint32)
    src = torch.from_numpy(rows.view(np.int32)).cuda()
    dst = torch.full_like(src, -1)
    golb200.rows_pass(src.data_ptr(), dst.data_ptr(), x, y, 4)
    torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy().view(np.uint32), oracle.life_rows(rows, x, 4, 32))


@pytest.mark.parametrize("x,y", SHAPES[1:4])
def test_run_vs_oracle(x, y):
    rows = np.random.default_rng(x).integers(0, 1 << 32, (y, x // 32), dtype=np.uint32)
    with golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32) as e:
        e.set_input_words(rows, 32)
        e.initialize_data_structures()
        assert e.plan()["temporal_steps"] == 4
        e.run(4 * 33 + 3)          # two chunks interleaved, a pass, a remainder
        e.run(130)
        e.finalize_data_structures()
        assert np.array_equal(e.fetch_words(32), oracle.life_rows(rows, x, 4 * 33 + 3 + 130, 32))
