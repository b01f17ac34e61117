"""The stand-alone PCG at the limits of its arguments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(rp, cols, vals, b, dtype, **kw):
    import torch

    import symx_gb300 as sg

    t = getattr(torch, dtype)
    x = torch.full((b.size,), float("nan"), dtype=t, device="cuda")
    info = sg.bcsr_pcg(torch.tensor(rp, device="cuda"), torch.tensor(cols, device="cuda"),
                       sg.component_major(torch.tensor(vals, dtype=t, device="cuda")),
                       torch.tensor(b, dtype=t, device="cuda"), x, **kw)
    return x.double().cpu().numpy(), info


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_exact_solution_converges_under_tolerances_whose_squares_underflow(lib, dtype):
    rp = np.arange(4, dtype=np.int32)
    x, info = _solve(rp, np.arange(3, dtype=np.int32), np.broadcast_to(np.eye(3) * 2.0, (3, 3, 3)).copy(), np.ones(9), dtype,
                     abs_tol=1e-200, rel_tol=1e-200)
    assert info["converged"] == 1 and info["found_indefiniteness"] == 0 and info["n_iterations"] == 1
    assert np.array_equal(x, np.full(9, 0.5))


def _laplace(n, band=40):
    i = np.concatenate([np.arange(n - 1), np.arange(n - band)])
    j = np.concatenate([np.arange(1, n), np.arange(band, n)])
    rows = np.concatenate([i, j, np.arange(n)])
    cols = np.concatenate([j, i, np.arange(n)])
    deg = np.bincount(i, minlength=n) + np.bincount(j, minlength=n)
    B = np.array([[1.0, 0.2, 0.0], [0.2, 1.0, 0.1], [0.0, 0.1, 1.0]])
    vals = np.concatenate([np.broadcast_to(-B, (2 * i.size, 3, 3)), np.eye(3) * (1.5 * deg + 0.5)[:, None, None]])
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return rp, cols[order].astype(np.int32), vals[order]


@pytest.mark.parametrize("dtype,power", [("float32", 60), ("float32", -50), ("float64", 480), ("float64", -480)])
def test_scaled_right_hand_side(lib, dtype, power):
    n = 30000  # b.b is beyond float's range at 2^60
    rp, cols, vals = _laplace(n)
    b = np.random.default_rng(5).uniform(0.5, 1.0, 3 * n).astype(dtype).astype(np.float64)
    x0, i0 = _solve(rp, cols, vals, b, dtype, abs_tol=0.0, rel_tol=1e-5)
    x, info = _solve(rp, cols, vals, b * 2.0 ** power, dtype, abs_tol=0.0, rel_tol=1e-5)
    assert i0["converged"] == 1 and info["converged"] == 1 and info["n_iterations"] == i0["n_iterations"]
    assert np.array_equal(x, x0 * 2.0 ** power)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("scale", [2.0 ** -20, 1.0, 2.0 ** 10])
def test_tight_relative_tolerances(lib, dtype, scale):
    """The recursive residual goes on falling below the rounding of b; 1e-22 of it is in range for any b."""
    n = 3000
    rp, cols, vals = _laplace(n)
    b = scale * np.random.default_rng(6).uniform(0.5, 1.0, 3 * n)
    for rel_tol in (1e-18, 1e-22):
        x, info = _solve(rp, cols, vals, b, dtype, abs_tol=0.0, rel_tol=rel_tol)
        assert info["converged"] == 1 and info["found_indefiniteness"] == 0
        assert info["error"] < rel_tol
