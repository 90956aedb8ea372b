"""Packed words in and out of an engine on the host: sizes around the copy's
64-byte steps, pages and threads, sources at any alignment. CPU only."""
import numpy as np
import pytest

import golb200


@pytest.mark.parametrize("words,y", [(1, 1), (1, 15), (1, 16), (1, 17), (3, 341), (5, 205), (32, 32),
                                     (33, 31), (157, 3001), (512, 4096), (511, 4099)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_words_in_and_out(words, y, offset):
    raw = np.random.default_rng(words * y).integers(0, 1 << 32, words * y + 8, dtype=np.uint32)
    rows = raw[offset:offset + words * y].reshape(y, words)
    with golb200.GolB200(grid_dimensions=(32 * words, y), state_bits_count=32) as e:
        e.set_input_words(rows, 32)
        assert np.array_equal(e.fetch_words(32), rows)
