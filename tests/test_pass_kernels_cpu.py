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


def test_refused():
    for args in ((64, 64, 17), (48, 64, 1), (96, 64, 2, 0, 4)):
        with pytest.raises(RuntimeError):
            golb200.rows_pass_kernel(*args)
