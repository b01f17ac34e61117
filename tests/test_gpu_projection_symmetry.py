"""The 12 x 12 projection writes both triangles of its result from one value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_12x12_results_are_symmetric(lib, dtype):
    import torch

    import symx_gb300 as sg

    rng = np.random.default_rng(3)
    A = rng.standard_normal((500, 12, 12))
    A = A + A.transpose(0, 2, 1)
    P = np.kron(np.eye(4) - 0.25, np.eye(3))
    A[::2] = (P @ A @ P)[::2]
    A = (0.5 * (A + A.transpose(0, 2, 1))).astype(dtype)
    got = torch.tensor(A, device="cuda")
    sg.project_pd(got, eps=1e-6)
    assert torch.equal(got, got.transpose(1, 2)) and not torch.equal(got.cpu(), torch.tensor(A))
