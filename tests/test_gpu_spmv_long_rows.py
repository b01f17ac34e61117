"""y = A x with rows of more than 24 blocks on average (in double by half a warp per row), around that
line and the rows of a thread block, with the reference and the bound of test_gpu_spmv_stream.py."""
import pytest

import test_gpu_spmv_stream as stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("lengths", [[24] * 33, [25] * 33, [27] * 70, [60] * 31, [200, 0, 30] * 11 + [1, 70], [300, 1],
                                     [24] * 32 + [25] * 32 + [3] * 9], ids=lambda v: f"{len(v)}rows_{sum(v)}")
def test_long_rows_match_float64(lib, dtype, lengths):
    stream.test_spmv_matches_float64(lib, dtype, lengths)
