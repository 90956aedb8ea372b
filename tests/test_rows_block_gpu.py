"""The register-block pass (gol_rows_pass without a forced band or lane width,
k >= 2) against the oracle: rows and columns at the edges of its blocks of
rows and of its 30-column warps, every depth, and grids of one block."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


def passed(cells, k):
    import torch
    y, x = cells.shape
    src = torch.from_numpy(oracle.pack_rows(cells, 32).view(np.int32)).cuda()
    dst = torch.full_like(src, -1)
    golb200.rows_pass(src.data_ptr(), dst.data_ptr(), x, y, k)
    torch.cuda.synchronize()
    return dst.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("k", [2, 3, 4, 5, 7, 8, 11, 12, 15, 16])
@pytest.mark.parametrize("words,y", [(1, 1), (1, 97), (2, 33), (28, 64), (29, 79), (30, 80),
                                     (31, 81), (59, 17), (60, 200), (61, 2), (157, 303),
                                     (330, 1001)])
def test_pass_vs_oracle(words, y, k):
    cells = oracle.random_ones_zeros(32 * words, y, words + y + k)
    want = oracle.pack_rows(oracle.life_cells(cells, k), 32)
    assert np.array_equal(passed(cells, k), want)


@pytest.mark.parametrize("x,y,gens", [(64, 40, 100), (1024, 1000, 333), (5024, 700, 97)])
def test_auto_engine_vs_oracle(x, y, gens):
    cells = oracle.random_ones_zeros(x, y, x + y)
    got = golb200.run_generations(cells, gens, state_bits_count=32)
    assert np.array_equal(got, oracle.life_cells(cells, gens))
