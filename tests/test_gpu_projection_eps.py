"""The projection with eps above eigenvalues that are positive, through project_pd and in the solver.

Tolerances, of max |H|: those of test_gpu_project_groups.py."""
import numpy as np
import pytest

from test_projection_accept import complement

pytestmark = pytest.mark.gpu
TOL = {"float32": 6e-5, "float64": 2.2e-13}


def _clamped(H, eps, mirroring):
    w, V = np.linalg.eigh(H)
    return np.einsum("eij,ej,ekj->eik", V, np.where(w < eps, -w if mirroring else eps, w), V)


@pytest.mark.parametrize("mirroring", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [12, 18, 24, 30])
def test_positive_eigenvalues_below_eps_are_clamped(lib, n, dtype, mirroring):
    """Translation-invariant matrices that are positive definite in the translations' complement, with
    eps between its smallest and its largest eigenvalue."""
    import torch

    import symx_gb300 as sg

    rng = np.random.default_rng(n)
    Q, m = complement(n), n - 3
    H = np.empty((300, n, n))
    for e in range(len(H)):
        V = np.linalg.qr(rng.standard_normal((m, m)))[0]
        w = rng.uniform(0.1, 1.0, m)
        w[0] = 0.01
        H[e] = Q @ (V * w) @ V.T @ Q.T
    H = (0.5 * (H + H.transpose(0, 2, 1))).astype(dtype)
    eps = float(np.dtype(dtype).type(0.05))
    got = torch.tensor(H, device="cuda")
    assert not sg.project_pd(got, eps=eps, mirroring=mirroring)
    ref = _clamped(H.astype(np.float64), eps, mirroring)
    err = np.abs(got.double().cpu().numpy() - ref).max(axis=(1, 2)) / np.abs(H).max(axis=(1, 2))
    assert err.max() <= TOL[dtype]


def test_solver_clamps_positive_eigenvalues_below_eps(lib):
    """The 12 x 12 projection of the mixed path (sorted and listed), with projection_eps inside the
    spectrum of most elements: no eigenvalue in the translations' complement stays below it."""
    import symx_gb300 as sg
    from symx_gb300 import problems

    p = problems.step_problem("tet4_6p")
    s = sg.ElasticSolver(p)
    s.set_settings(precision="mixed")
    s.set_state(p["x_init"], p["x0"], p["v0"])
    _, _, H = s.element_outputs(0, project=False)
    Q = complement(12)
    eps = float(np.median(np.linalg.eigvalsh(Q.T @ H @ Q)))
    s.set_settings(projection_eps=eps)
    _, _, P = s.element_outputs(0, project=True)
    w, V = np.linalg.eigh(Q.T @ H @ Q)
    assert np.count_nonzero((w[:, 0] > 0) & (w[:, 0] < eps)) > 10
    ref = np.einsum("eij,ej,ekj->eik", V, np.maximum(w, eps), V)
    assert np.abs(Q.T @ P @ Q - ref).max() <= TOL["float32"] * np.abs(H).max()
