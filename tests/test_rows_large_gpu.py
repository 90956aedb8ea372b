"""Depths 2 to 4 just below and above the size at which whole-lane grids take
the K-stage pipeline: the same words as that many one-generation passes."""
import pytest

import golb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 3, 4])
@pytest.mark.parametrize("words,rows", [(1024, 16384), (1024, 16385), (1023, 16500), (4100, 4100),
                                        (512, 33000), (256, 65536), (256, 65537)])
def test_equals_single_passes(words, rows, k):
    import torch
    torch.manual_seed(words + k)
    src = torch.randint(-2**31, 2**31 - 1, (rows, words), dtype=torch.int32, device="cuda")
    got = torch.full_like(src, -1)
    golb200.rows_pass(src.data_ptr(), got.data_ptr(), 32 * words, rows, k)
    a, b = src.clone(), torch.empty_like(src)
    for _ in range(k):
        golb200.rows_pass(a.data_ptr(), b.data_ptr(), 32 * words, rows, 1)
        a, b = b, a
    torch.cuda.synchronize()
    assert torch.equal(got, a)
