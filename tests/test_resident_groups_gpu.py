"""Resident runs at the widths and band heights where their row groups change,
against the oracle: generations within an epoch, whole epochs and a rest."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu

LANES = (3, 7, 8, 12, 13, 15, 16, 17, 31, 32, 47, 48, 63, 64, 65, 80, 81, 88, 96, 112, 113, 128, 256)


@pytest.mark.parametrize("lanes", LANES)
@pytest.mark.parametrize("y", [24, 148 * 8 + 3, 148 * 21, 148 * 29, 148 * 41])
def test_resident_vs_oracle(lanes, y):
    for words in (4 * lanes, 4 * lanes - 2):
        row = (words // 2 + 31) // 32 * 64 + 8          # a row as the limit counts it
        if 2 * (-(-y // min(148, y // 8)) + 16) * row * 4 + 1024 > 227 * 1024:
            pytest.skip("does not fit")
        rows = np.random.default_rng(words + y).integers(0, 1 << 32, (y, words), dtype=np.uint32)
        with golb200.GolB200(grid_dimensions=(32 * words, y), state_bits_count=32,
                             algorithm="resident") as e:
            e.set_input_words(rows, 32)
            e.initialize_data_structures()
            e.run(21)
            e.run(8)
            e.finalize_data_structures()
            assert np.array_equal(e.fetch_words(32), oracle.life_rows(rows, 32 * words, 29, 32))
