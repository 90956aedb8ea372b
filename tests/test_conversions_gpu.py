"""Device conversions at the shapes their kernels branch on: rows of one to
five words, row groups cut short, buffers off the 16-byte boundary, and byte
cells of any nonzero value."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("layout,bits", [(l, b) for l in ("columns", "tiles") for b in (16, 32, 64)])
@pytest.mark.parametrize("x", [32, 64, 96, 128, 160, 4096 + 32])
@pytest.mark.parametrize("offset", [0, 8])
def test_layouts(layout, bits, x, offset):
    yb = golb200.layout_block(layout, bits)[1]
    for y in (yb, 3 * yb, 64 + yb):
        g = oracle.random_ones_zeros(x, y, x + y)
        want = oracle.pack_layout(g, golb200.LAYOUTS[layout], bits)
        n = x * y // 32
        src = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
        dst, back = torch.full_like(src, 7), torch.full_like(src, 7)
        o = offset // 4
        src[o:o + n] = torch.from_numpy(oracle.pack_rows(g, 32).view(np.int32).reshape(-1)).cuda()
        golb200.rows_to_layout_device(src[o:].data_ptr(), dst[o:].data_ptr(), x, y, layout, bits)
        golb200.layout_to_rows_device(dst[o:].data_ptr(), back[o:].data_ptr(), x, y, layout, bits)
        torch.cuda.synchronize()
        assert dst[o:o + n].cpu().numpy().tobytes() == want.tobytes(), (x, y)
        assert torch.equal(back[o:o + n], src[o:o + n]), (x, y)
        assert (dst[:o] == 7).all() and (dst[o + n:] == 7).all()
        assert (back[:o] == 7).all() and (back[o + n:] == 7).all()


@pytest.mark.parametrize("x,y", [(32, 1), (32, 7), (96, 33), (2048, 4097), (16384, 130)])
def test_cells(x, y):
    rng = np.random.default_rng(x + y)
    cells = rng.integers(0, 256, (y, x), dtype=np.uint8) * rng.integers(0, 2, (y, x), dtype=np.uint8)
    want = oracle.pack_rows((cells != 0).astype(np.uint8), 32).view(np.int32)
    c = torch.from_numpy(cells).cuda()
    w = torch.full((y, x // 32), -1, dtype=torch.int32, device="cuda")
    back = torch.full_like(c, 9)
    golb200.pack_cells_device(c.data_ptr(), w.data_ptr(), x, y)
    golb200.unpack_cells_device(w.data_ptr(), back.data_ptr(), x, y)
    torch.cuda.synchronize()
    assert np.array_equal(w.cpu().numpy(), want)
    assert np.array_equal(back.cpu().numpy(), (cells != 0).astype(np.uint8))
