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
