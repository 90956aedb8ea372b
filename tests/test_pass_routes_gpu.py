"""Large passes that the K-stage pipeline takes at widths other than powers of
two, against passes of one generation, on grids with live rows at every edge."""
import pytest

import golb200

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,k", [(32640, 16481, 2), (65024, 8261, 2), (4096, 122881, 3),
                                   (7936, 50801, 4), (3840, 104859, 4), (4096, 131073, 6),
                                   (4096, 131073, 7), (8192, 65537, 8)])
def test_pass_equals_single_generations(x, y, k):
    assert golb200.rows_pass_kernel(x, y, k).startswith("rows_temporal")
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    a = torch.randint(-(1 << 31), 1 << 31, (y, x // 32), dtype=torch.int32, device="cuda", generator=g)
    src, out = a.clone(), torch.empty_like(a)
    s = torch.cuda.current_stream().cuda_stream
    golb200.rows_pass(src.data_ptr(), out.data_ptr(), x, y, k, stream=s)
    b = torch.empty_like(a)
    for _ in range(k):
        golb200.rows_pass(a.data_ptr(), b.data_ptr(), x, y, 1, stream=s)
        a, b = b, a
    torch.cuda.synchronize()
    assert torch.equal(out, a)
