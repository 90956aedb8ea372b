"""The row-pair pipeline on rows wider than a CTA: x-slices with a halo lane
each side, rows as they are and interleaved in a run, against passes of one
generation. Heights around bands, live cells at the slices' seams."""
import pytest

import golb200

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def random_words(x, y, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-(1 << 31), 1 << 31, (y, x // 32), dtype=torch.int32, device="cuda", generator=g)


def single_generations(a, x, y, n):
    s = torch.cuda.current_stream().cuda_stream
    a, b = a.clone(), torch.empty_like(a)
    for _ in range(n):
        golb200.rows_pass(a.data_ptr(), b.data_ptr(), x, y, 1, stream=s)
        a, b = b, a
    torch.cuda.synchronize()
    return a


SHAPES = [(65024, 8192), (65024, 8191), (64512, 8300), (97536, 6001), (130048, 4150)]


@pytest.mark.parametrize("x,y", SHAPES)
def test_pass(x, y):
    assert golb200.rows_pass_kernel(x, y, 4) == "rows_pair_kernel<4>"
    src = random_words(x, y, x + y)
    out = torch.full_like(src, -1)
    golb200.rows_pass(src.data_ptr(), out.data_ptr(), x, y, 4, stream=torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out, single_generations(src, x, y, 4))


@pytest.mark.parametrize("x,y", SHAPES[:3])
def test_run(x, y):
    assert golb200.rows_pass_kernel(x, y, 4) == "rows_pair_kernel<4>"
    src = random_words(x, y, x - y)
    gens = 4 * 33 + 3          # two chunks of interleaved rows, a pass and a rest
    with golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32) as e:
        e.set_input_words(src.cpu().numpy().view("uint32"), 32)
        e.initialize_data_structures()
        assert e.plan()["temporal_steps"] == 4
        e.run(gens)
        e.finalize_data_structures()
        got = torch.from_numpy(e.fetch_words(32).view("int32")).cuda()
    assert torch.equal(got, single_generations(src, x, y, gens))


@pytest.mark.parametrize("x,y", [(16384, 16384), (16384, 16001), (16000, 17003), (32768, 16386)])
def test_unsliced_shapes_run_it_too(x, y):
    assert golb200.rows_pass_kernel(x, y, 4) == "rows_pair_kernel<4>"
