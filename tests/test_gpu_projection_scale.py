"""The projection of double matrices that are zero, or nearly, beside eps.

Tolerance, of eps: that of test_gpu_project_groups.py."""
import numpy as np
import pytest

from test_projection_accept import complement

pytestmark = pytest.mark.gpu
TOL = 2.2e-13


def _clamped(H, eps):
    w, V = np.linalg.eigh(H)
    return np.einsum("eij,ej,ekj->eik", V, np.maximum(w, eps), V)


@pytest.mark.parametrize("eps", [1e-10, 1.0, 1e9, 1e300])
@pytest.mark.parametrize("n", [12, 18, 24, 30])
def test_eps_far_above_the_matrix(lib, n, eps):
    import torch

    import symx_gb300 as sg

    H = np.zeros((3, n, n))
    H[1] = complement(n) @ complement(n).T * 1e-280
    H[2] = -np.eye(n) * 1e-12
    got = torch.tensor(H, device="cuda")
    assert not sg.project_pd(got, eps=eps)
    ref = _clamped(H, eps)
    assert np.abs(got.cpu().numpy() / eps - ref / eps).max() <= TOL
