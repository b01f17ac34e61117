"""The projection of double matrices leaves one as it is only when every eigenvalue in the complement
of the rigid translations is positive, however small the negative ones are: 12 x 12 on the host, all
sizes on the GPU against numpy's eigh.

GPU tolerance, of max |H|: that of test_gpu_project_groups.py (2.2e-13)."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def complement(n):
    """Orthonormal basis of the node space orthogonal to the rigid translations."""
    k = n // 3
    B = np.zeros((k, k - 1))
    for m in range(1, k):
        B[:m, m - 1] = 1.0 / np.sqrt(m * (m + 1))
        B[m, m - 1] = -m / np.sqrt(m * (m + 1))
    return np.kron(B, np.eye(3))


def nearly_definite(n, count, seed, negative=True):
    """Translation-invariant matrices of size about one whose complement has one eigenvalue of size
    1e-12 .. 1e-6 (of that sign) and the others in 1e-4 .. 1: random eigenvectors, and for every second
    matrix those of a graded one, where a factorization's last pivot is far from the eigenvalue."""
    rng = np.random.default_rng(seed)
    Q, m = complement(n), n - 3
    out = np.empty((count, n, n))
    for e in range(count):
        w = 10.0 ** rng.uniform(-4, 0, m)
        w[0] = (-1.0 if negative else 1.0) * 10.0 ** rng.uniform(-12, -6)
        V = np.linalg.qr(rng.standard_normal((m, m)))[0]
        B = (V * w) @ V.T
        if e % 2:
            L = np.tril(rng.standard_normal((m, m)) * 10.0 ** rng.uniform(-1, 0.5, (m, 1)), -1) + np.eye(m)
            B = (L * np.abs(w)) @ L.T
            u, U = np.linalg.eigh(B / np.abs(B).max())
            u[1:] = np.maximum(u[1:], 1e-4)
            u[0] = w[0]
            B = (U * u) @ U.T
        out[e] = Q @ B @ Q.T
    return 0.5 * (out + out.transpose(0, 2, 1))


def test_host_accepts_only_definite_matrices(tmp_path):
    exe = tmp_path / "accept"
    subprocess.run(["g++", "-std=c++17", "-O2", os.path.join(ROOT, "tests", "cpp", "test_projection_accept_host.cpp"),
                    "-o", str(exe)], check=True)
    bad = nearly_definite(12, 20000, seed=1)
    Q = complement(12)
    good = nearly_definite(12, 500, seed=2, negative=False)
    good += Q @ Q.T * 1e-4  # smallest eigenvalue 1e-4
    H = np.concatenate([bad, good])
    (tmp_path / "in").write_bytes(np.int64(len(H)).tobytes() + H.tobytes())
    subprocess.run([str(exe), str(tmp_path / "in"), str(tmp_path / "out")], check=True)
    got = np.frombuffer((tmp_path / "out").read_bytes(), np.int32).reshape(2, -1)
    assert np.array_equal(got[0], got[1])
    assert np.all(got[0][:len(bad)] == 1)
    assert np.all(got[0][len(bad):] == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("mirroring", [False, True])
@pytest.mark.parametrize("n", [12, 18, 24, 30])
def test_small_negative_eigenvalues_are_clamped(lib, n, mirroring):
    import torch

    import symx_gb300 as sg

    eps = 1e-10
    H = nearly_definite(n, 2000, seed=n)
    got = torch.tensor(H, device="cuda")
    assert not sg.project_pd(got, eps=eps, mirroring=mirroring)
    w, V = np.linalg.eigh(H)
    ref = np.einsum("eij,ej,ekj->eik", V, np.where(w < eps, -w if mirroring else eps, w), V)
    err = np.abs(got.cpu().numpy() - ref).max(axis=(1, 2)) / np.abs(H).max(axis=(1, 2))
    assert err.max() <= 2.2e-13
