"""One-generation passes without a forced band (bands loaded whole): word
counts for every lane width around a warp's and a CTA's ends, rows around a
band's."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [1, 2, 3, 4, 31, 32, 33, 62, 64, 66, 65, 124, 128, 132, 252, 256,
                                   260, 513])
@pytest.mark.parametrize("wpl", [0, 1, 2, 4])
def test_vs_oracle(words, wpl):
    import torch
    if wpl and words % wpl:
        pytest.skip("rows are not whole lanes")
    for y in (1, 2, 15, 16, 17, 30, 31, 33, 100):
        rows = np.random.default_rng(words + y).integers(0, 1 << 32, (y, words), dtype=np.uint32)
        src = torch.from_numpy(rows.view(np.int32)).cuda()
        dst = torch.full_like(src, -1)
        golb200.rows_pass(src.data_ptr(), dst.data_ptr(), 32 * words, y, 1, lane_words=wpl)
        torch.cuda.synchronize()
        want = oracle.life_rows(rows, 32 * words, 1, 32)
        assert np.array_equal(dst.cpu().numpy().view(np.uint32), want), y
