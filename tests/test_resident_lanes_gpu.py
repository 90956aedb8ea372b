"""Resident runs and batches at the widths where the interleaved rows change:
one to nine words (whole and partial lanes of four), odd word counts, rows
whose lanes do not fill warps, bands of K rows and single bands."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu

SHAPES = [(w, y) for w in (1, 2, 3, 4, 5, 7, 8, 9) for y in (1, 9, 70)] + \
         [(31, 300), (33, 64), (129, 257), (157, 500), (255, 161), (509, 40), (1021 - 1, 33)]


def accepted(words, y, k):
    """The limit of a resident run on a B200 (148 SMs, 227 KB each)."""
    unit = 2 - words % 2
    lanes = -(-words // unit // 32) * 32
    bands = max(1, min(148, y // k))
    rows = -(-y // bands) + 2 * k
    return lanes <= 512 and 2 * rows * (lanes * unit + 8) * 4 + 1024 <= 227 * 1024


@pytest.mark.parametrize("words,y", SHAPES)
@pytest.mark.parametrize("k", [0, 1, 3, 16])
def test_resident_vs_oracle(words, y, k):
    cells = oracle.random_ones_zeros(32 * words, y, words + y + k)
    if not accepted(words, y, k or 8):
        with pytest.raises(RuntimeError):
            golb200.run_generations(cells, 1, algorithm="resident", temporal_steps=k,
                                    state_bits_count=32)
        return
    for gens in (1, 37):
        got = golb200.run_generations(cells, gens, algorithm="resident", temporal_steps=k,
                                      state_bits_count=32)
        assert np.array_equal(got, oracle.life_cells(cells, gens)), gens


def test_resident_batch_vs_oracle():
    work = [(oracle.random_ones_zeros(32 * w, y, w + y), 5 + (w * y) % 60) for w, y in SHAPES]
    with golb200.GolBatch() as b:
        ids = [b.add(c, n) for c, n in work]
        for _ in range(2):
            b.run_resident()
            b.sync()
            for gid, (c, n) in zip(ids, work):
                assert np.array_equal(b.fetch(gid), oracle.life_cells(c, n)), (c.shape, n)


@pytest.mark.parametrize("words,y,ok", [(1024, 64, True), (1026, 64, False), (511, 64, True),
                                        (513, 64, False), (1, 148 * 690, True),
                                        (1, 148 * 710, False), (5, 148 * 710, False)])
def test_refusals_stay(words, y, ok):
    """The grids a resident run takes and refuses: rows of up to 1024 words (512
    when odd), bands that fit with rows padded as the limit counts them."""
    with golb200.GolB200(grid_dimensions=(32 * words, y), state_bits_count=32,
                         algorithm="resident") as e:
        e.set_input_words(np.zeros((y, words), np.uint32), 32)
        if ok:
            e.initialize_data_structures()
        else:
            with pytest.raises(RuntimeError):
                e.initialize_data_structures()
