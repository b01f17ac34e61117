"""Projection by a group of lanes per matrix (project_warp.cu) against numpy's eigh, through
symxg_project_pd_*: counts around a tile and a warp's groups, translation-invariant and general
matrices mixed (positive definite, indefinite, degenerate, zero), and scales far from one.

Tolerance, of max |H|: the Jacobi iterations stop at off-diagonal entries of 2^-19 (float) and
2^-48 (double) of it, at most n of them in a row: n 2^-19 = 5.7e-5 and n 2^-48 + n^2 u = 2.1e-13
at n = 30.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"float32": 6e-5, "float64": 2.2e-13}


def _reference(H, eps, mirroring):
    """Clamped eigenvalues; a matrix that is positive definite in the complement of the rigid
    translations is left as it is (its translations' eigenvalues are not lifted to eps)."""
    n = H.shape[1]
    w, V = np.linalg.eigh(H)
    clamped = np.where(w < eps, -w if mirroring else eps, w)
    size = np.abs(H).max(axis=(1, 2))
    rigid = np.abs(H @ np.kron(np.ones((n // 3, 1)), np.eye(3))).max(axis=(1, 2)) <= 1e-5 * size
    done = rigid & (size > 0) & (w[:, 3] > 1e-4 * size)
    return np.where(done[:, None, None], H, np.einsum("eij,ej,ekj->eik", V, clamped, V))


def _matrices(n, count, seed):
    """A mix of kinds, cycled over the matrices so that neighbouring lanes and groups differ."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((count, n, n))
    A = A + A.transpose(0, 2, 1)
    k = n // 3
    P = np.kron(np.eye(k) - 1.0 / k, np.eye(3))  # removes the rigid translations
    kind = np.arange(count) % 7
    inv = P @ A @ P
    psd = P @ (A @ A) @ P
    out = np.where((kind == 0)[:, None, None], A, inv)  # 0: general indefinite, 1: invariant indefinite
    out[kind == 2] = psd[kind == 2]  # invariant, positive definite in the complement
    out[kind == 3] = 0.0
    q = np.linalg.qr(P @ A)[0]  # degenerate: two eigenvalues only
    two = np.einsum("eij,j,ekj->eik", q, np.where(np.arange(n) < n // 2, 1.0, -1.0), q)
    out[kind == 4] = (P @ two @ P)[kind == 4]
    out[kind == 5] = np.einsum("eij,ekj->eik", A, A)[kind == 5]  # general, positive definite
    out[kind == 6] *= 10.0 ** rng.uniform(-12, 12, count)[kind == 6][:, None, None]
    return 0.5 * (out + out.transpose(0, 2, 1))


@pytest.mark.parametrize("mirroring", [False, True])
@pytest.mark.parametrize("n,dtype,count", [(12, "float64", 1), (12, "float64", 7), (12, "float64", 129),
                                           (12, "float64", 3001), (12, "float32", 1), (12, "float32", 33),
                                           (12, "float32", 1500), (18, "float32", 33), (18, "float64", 33),
                                           (24, "float32", 9), (24, "float64", 141), (30, "float32", 141),
                                           (30, "float64", 15)])
def test_projection_matches_eigh(lib, n, dtype, count, mirroring):
    import torch

    import symx_gb300 as sg

    eps = 1e-6
    H = _matrices(n, count, seed=n + count).astype(dtype)
    got = torch.tensor(H, device="cuda")
    assert not sg.project_pd(got, eps=eps, mirroring=mirroring)
    ref = _reference(H.astype(np.float64), np.dtype(dtype).type(eps).astype(np.float64), mirroring)
    scale = np.maximum(np.abs(H).max(axis=(1, 2)).astype(np.float64), eps)
    err = np.abs(got.double().cpu().numpy() - ref).max(axis=(1, 2)) / scale
    assert np.max(err) <= TOL[dtype], (int(np.argmax(err)) % 7, np.max(err))


def test_extreme_scales_and_nan(lib):
    import torch

    import symx_gb300 as sg

    base = _matrices(12, 7, seed=1)[1]
    for n, dtype, s in ((12, "float64", 1e200), (12, "float64", 1e-200), (24, "float64", 1e150)):
        A = base if n == 12 else _matrices(24, 7, seed=2)[1]
        H = (A * s).astype(dtype)
        got = torch.tensor(H[None], device="cuda")
        assert not sg.project_pd(got, eps=1e-3 * s)
        ref = _reference(A[None], 1e-3, False)
        assert np.max(np.abs(got.cpu().numpy() / s - ref)) <= TOL[dtype] * np.abs(A).max()
    for n in (12, 24):  # a NaN matrix does not spread to its neighbours
        H = _matrices(n, 6, seed=3)
        H[2] = np.nan
        got = torch.tensor(H, device="cuda")
        sg.project_pd(got, eps=1e-6)
        keep = np.arange(6) != 2
        ref = _reference(H[keep], 1e-6, False)
        assert np.max(np.abs(got.cpu().numpy()[keep] - ref)) <= TOL["float64"] * np.abs(H[keep]).max()


@pytest.mark.parametrize("n,dtype", [(12, "float32"), (12, "float64"), (18, "float32"), (24, "float64"), (30, "float32")])
def test_contiguous_and_strided_matrices_agree(lib, n, dtype):
    """Contiguous matrices are projected where they lie, others through a block-major copy: the
    same operations, so the same bits; views that share the storage see the result."""
    import torch

    import symx_gb300 as sg

    H = torch.tensor(_matrices(n, 97, seed=5).astype(dtype), device="cuda")
    rows, wide = H.clone(), torch.zeros(97, n, 2 * n, dtype=H.dtype, device="cuda")
    wide[:, :, :n] = H
    sg.project_pd(rows, eps=1e-6)
    sg.project_pd(wide[:, :, :n], eps=1e-6)
    assert torch.equal(rows, wide[:, :, :n]) and not torch.equal(rows, H)
    assert not wide[:, :, n:].any()
    shifted = torch.zeros(H.numel() + 1, dtype=H.dtype, device="cuda")  # not 16-byte aligned
    shifted[1:] = H.flatten()
    sg.project_pd(shifted[1:].view_as(H), eps=1e-6)
    assert torch.equal(shifted[1:].view_as(H), rows) and shifted[0] == 0


def test_autograd_sees_the_projection(lib):
    import torch

    import symx_gb300 as sg

    H = torch.tensor(_matrices(12, 7, seed=6), device="cuda")
    version = H._version
    sg.project_pd(H)
    assert H._version > version
    leaf = H.clone().requires_grad_()
    with pytest.raises(RuntimeError):
        sg.project_pd(leaf)


@pytest.mark.parametrize("dtype,copies", [("float32", 4800), ("float64", 600)])
def test_more_matrices_than_one_pass_of_tiles(lib, dtype, copies):
    """Several tiles per block; and each matrix's bits do not depend on those next to it."""
    import torch

    import symx_gb300 as sg

    H = torch.tensor(_matrices(12, 101, seed=8).astype(dtype), device="cuda")
    few = H.clone()
    sg.project_pd(few, eps=1e-6)
    many = H.repeat(copies, 1, 1)
    sg.project_pd(many, eps=1e-6)
    assert torch.equal(many, few.repeat(copies, 1, 1))
