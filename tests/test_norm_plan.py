"""The rule that gives a row of a norm a thread block or warps, on the CPU, against times measured on a B200 with either forced (microseconds
of norm + quantise)."""
import ctypes

import pytest

# (rows, columns, block per row, warps per row)
MEASURED = [
    (1023, 1024, 3.0, 3.8), (2895, 512, 4.0, 3.0), (1447, 2048, 4.6, 5.8), (681, 3072, 3.6, 4.3), (964, 3072, 4.7, 4.4), (511, 4096, 3.7, 4.7),
    (455, 4608, 4.93, 4.57), (372, 5632, 5.03, 4.91), (297, 6144, 4.54, 4.32), (341, 6144, 5.22, 4.61), (255, 8192, 3.9, 5.1), (361, 8192, 5.5, 5.3),
]


@pytest.mark.parametrize("rows,cols,block_us,warps_us", MEASURED)
def test_takes_the_faster_kernel(rows, cols, block_us, warps_us):
    from train_gpt_b200 import build, _lib
    build.build()
    few = _lib.load().tgh_norm_few_rows(ctypes.c_int64(rows), ctypes.c_int64(cols))
    assert (block_us if few else warps_us) <= 1.02 * min(block_us, warps_us)
