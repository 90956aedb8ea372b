"""Which kernel a pass runs, by size, depth and forced band or lane width, as
the planner says it (148 SMs, as on a B200). CPU only."""
import pytest

import golb200


@pytest.mark.parametrize("x,y,k,band,lanes,kernel", [
    (32768, 32768, 1, 0, 0, "rows_once_kernel<4>"),
    (32768, 32768, 1, 9, 0, "rows_stream_kernel<4>"),
    (32768, 32768, 2, 0, 0, "rows_temporal_kernel<4,2>"),
    (32768, 32768, 3, 0, 0, "rows_temporal_kernel<4,3>"),
    (16384, 16384, 4, 0, 0, "rows_pair_kernel<4>"),
    (16384, 16384, 8, 0, 0, "rows_block_kernel<96>"),
    (16384, 16384, 8, 0, 2, "rows_temporal_kernel<2,8>"),
    (16384, 16384, 4, 32, 0, "rows_temporal_kernel<4,4>"),
])
def test_kernel_by_name(x, y, k, band, lanes, kernel):
    assert golb200.rows_pass_kernel(x, y, k, band, lanes) == kernel


@pytest.mark.parametrize("x,y,k,kernel", [
    # large grids next to 32768 and 8192 cells wide, where the K-stage pipeline
    # is the faster form too
    (32640, 32768, 2, "rows_temporal_kernel<4,2>"),
    (30720, 32768, 2, "rows_temporal_kernel<4,2>"),
    (32640, 32768, 3, "rows_temporal_kernel<4,3>"),
    (65024, 16384, 2, "rows_temporal_kernel<4,2>"),
    (8192, 65536, 4, "rows_temporal_kernel<4,4>"),
    (7936, 67650, 4, "rows_temporal_kernel<4,4>"),
    (3840, 200000, 4, "rows_temporal_kernel<4,4>"),
    (4096, 262144, 7, "rows_temporal_kernel<2,7>"),
    # and where it is not: warps that do not share the SMs evenly, idle lanes, L2
    (20480, 32768, 2, "rows_block"),
    (18432, 32768, 3, "rows_block"),
    (33280, 32768, 2, "rows_block"),
    (6144, 131072, 4, "rows_block"),
    (16384, 12288, 2, "rows_block"),
])
def test_large_grids(x, y, k, kernel):
    got = golb200.rows_pass_kernel(x, y, k)
    if kernel == "rows_block":
        assert got.startswith(kernel)
    else:
        assert got == kernel


def test_refused():
    for args in ((64, 64, 17), (48, 64, 1), (96, 64, 2, 0, 4)):
        with pytest.raises(RuntimeError):
            golb200.rows_pass_kernel(*args)
