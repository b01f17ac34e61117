"""The PCG kernels behind k_pcg_resident: the staged one-launch kernel (the mixed solver above about
145,000 block rows or 110 MB of matrix values, or with an option of its own) and the two launches per
iteration (FP64, and the stand-alone solve, above about 80,000 rows in double and 145,000 in float).

Tolerances: positions of a mixed solve within 1e-6 of the displacement of the FP64 one, as
test_gpu_parity.py; true residuals within 10 x rel_tol, as test_gpu_pcg.py."""
import numpy as np
import pytest

from test_gpu_pcg_resident import _spd

pytestmark = pytest.mark.gpu


def _solve(p, **settings):
    import symx_gb300 as sg

    s = sg.ElasticSolver(p)
    s.set_settings(cg_rel_tolerance=1e-3, **settings)
    s.set_state(p["x_init"], p["x0"], p["v0"])
    st = s.solve()
    assert st["solver_return"] == 0
    return s, st, s.get_positions()


def test_staged_waits_give_up(lib):
    """As test_gpu_failure.py has it for the kernel that small systems take without an option."""
    import symx_gb300 as sg
    from symx_gb300 import problems

    p = problems.step_problem("tet4_6p")
    s, ref, x_ref = _solve(p, precision="mixed", cg_fp64_partial_sums=1)
    lib.symxg_set_wait_poll_limit(0)
    try:
        s.set_state(p["x_init"], p["x0"], p["v0"])
        with pytest.raises(sg.SymxgError, match="bounded wait"):
            s.solve()
    finally:
        lib.symxg_set_wait_poll_limit(-1)
    s.set_state(p["x_init"], p["x0"], p["v0"])
    assert s.solve()["cg_iterations"] == ref["cg_iterations"] and np.array_equal(s.get_positions(), x_ref)


@pytest.mark.parametrize("case", ["tet4_6p", "tet4_10", "hex8_3"])
def test_look_ahead_matches_reference(lib, golden, case):
    from symx_gb300 import problems

    p = problems.step_problem(case)
    _, st, x = _solve(p, precision="mixed", cg_lookahead=1)
    sol = golden(f"{case}_solve")
    assert st["newton_iterations"] == int(sol["newton_iterations_full"])
    assert np.linalg.norm(x - sol["x_full"]) / np.linalg.norm(sol["x_full"] - p["x0"]) < 1e-6


@pytest.mark.parametrize("kind,cells", [("tet4", (53, 53, 53)), ("hex8", (50, 50, 50))])
def test_systems_beyond_the_resident_kernel(lib, kind, cells):
    """157,464 rows (neither precision resident) and 132,651 rows of 27 blocks (the mixed values exceed
    13/16 of L2): the staged kernel in its default form against two FP64 launches per iteration."""
    from symx_gb300 import problems

    cfg = {"kind": kind, "cells": cells, "h": 0.01, "perturb": 0.05, "seed": 3}
    if kind == "hex8":
        cfg.update(perturb=0.0, youngs_lognormal_sigma=0.5)
    p = problems.step_problem(cfg, youngs=1e5, poisson=0.3, density=1000.0, dt=1.0 / 60.0, k_bc=1e8)
    _, st, x = _solve(p, precision="mixed")
    _, ref, x_ref = _solve(p, precision="fp64")
    assert st["newton_iterations"] == ref["newton_iterations"]
    assert np.linalg.norm(x - x_ref) / np.linalg.norm(x_ref - p["x0"].reshape(x_ref.shape)) < 1e-6


@pytest.mark.parametrize("dtype,n,rel_tol", [("float32", 150001, 1e-5), ("float64", 90001, 1e-9)])
def test_stand_alone_two_launch_residual(lib, dtype, n, rel_tol):
    import scipy.sparse as sp
    import torch

    import symx_gb300 as sg

    rp, cols, vals = _spd(n, (1, 2, 50, 51, 2500, 2551, 2552), 0, seed=n)
    t = getattr(torch, dtype)
    vals = torch.tensor(vals, dtype=t)
    b = torch.tensor(np.random.default_rng(n).standard_normal(3 * n), dtype=t)
    x = torch.full((3 * n,), float("nan"), dtype=t, device="cuda")
    info = sg.bcsr_pcg(torch.tensor(rp, device="cuda"), torch.tensor(cols, device="cuda"), sg.component_major(vals.cuda()),
                       b.cuda(), x, rel_tol=rel_tol, abs_tol=1e-14)
    assert info["converged"] == 1 and info["found_indefiniteness"] == 0
    r = b.double().numpy() - sp.bsr_matrix((vals.double().numpy(), cols, rp), shape=(3 * n, 3 * n)) @ x.double().cpu().numpy()
    assert np.linalg.norm(r) <= 10 * rel_tol * np.linalg.norm(b.double().numpy())
