"""k_pcg_resident with rows of more than 80 blocks (16 lanes per row, several rounds per block), with the
reference and the tolerance of test_gpu_pcg_resident.py."""
import pytest

import test_gpu_pcg_resident as resident

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,rel_tol", [("float32", 1e-5), ("float64", 1e-9)])
@pytest.mark.parametrize("n", [9001, 13001])
def test_long_rows(lib, n, dtype, rel_tol):
    resident.test_true_residual(lib, n, tuple(range(1, 46)), 0, dtype, rel_tol)
