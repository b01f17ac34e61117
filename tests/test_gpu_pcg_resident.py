"""One-launch PCG with the matrix in shared memory (k_pcg_resident) at the edges of its layouts,
through symxg_bcsr_pcg_*: one block and a grid, row counts around a block's minimum share, both
lane counts per row, rows that stay in global memory, and a gather list that does not fit
(random columns in double), against the true residual in float64.

Tolerance: the recursive residual reaches rel_tol; the true one |b - A x| / |b| follows it to
rounding on these well-conditioned systems, so 10 x rel_tol (the bound of test_gpu_pcg.py).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, offsets, per_row, seed):
    """Symmetric block matrix: blocks at the given column offsets, or `per_row` random columns per
    row, and a diagonal block that dominates its row."""
    rng = np.random.default_rng(seed)
    if per_row:
        i = np.repeat(np.arange(n), per_row // 2)
        j = rng.integers(0, n, i.size)
    else:
        i = np.concatenate([np.arange(n - o) for o in offsets if o < n] or [np.zeros(0, int)])
        j = np.concatenate([np.arange(o, n) for o in offsets if o < n] or [np.zeros(0, int)])
    keep = i != j
    key = np.unique(np.minimum(i, j)[keep].astype(np.int64) * n + np.maximum(i, j)[keep])
    i, j = key // n, key % n
    B = rng.standard_normal((i.size, 3, 3)) / 6.0
    deg = np.bincount(i, minlength=n) + np.bincount(j, minlength=n)
    D = np.eye(3) * (1.0 + deg)[:, None, None]
    rows = np.concatenate([i, j, np.arange(n)])
    cols = np.concatenate([j, i, np.arange(n)])
    vals = np.concatenate([B, B.transpose(0, 2, 1), D])
    order = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return rp.astype(np.int32), cols[order].astype(np.int32), vals[order]


@pytest.mark.parametrize("dtype,rel_tol", [("float32", 1e-5), ("float64", 1e-9)])
@pytest.mark.parametrize("n,offsets,per_row", [(1, (), 0), (15, (1, 2), 0), (17, (1, 5), 0), (239, (1, 7, 8), 0),
                                               (2433, (1, 40, 41, 1200), 0), (9721, (1, 21, 22, 441, 462), 0),
                                               (40001, (1, 2, 33, 34, 1089, 1122, 1123), 0), (20000, (), 60)])
def test_true_residual(lib, n, offsets, per_row, dtype, rel_tol):
    import scipy.sparse as sp
    import torch

    import symx_gb300 as sg

    rp, cols, vals = _spd(n, offsets, per_row, seed=n)
    t = getattr(torch, dtype)
    vals = torch.tensor(vals, dtype=t)
    b = torch.tensor(np.random.default_rng(n + 1).standard_normal(3 * n), dtype=t)
    x = torch.full((3 * n,), float("nan"), dtype=t, device="cuda")
    A = sp.bsr_matrix((vals.double().numpy(), cols, rp), shape=(3 * n, 3 * n))
    for _ in range(2):  # a second solve in the same workspace addresses
        x.fill_(float("nan"))
        info = sg.bcsr_pcg(torch.tensor(rp, device="cuda"), torch.tensor(cols, device="cuda"),
                           sg.component_major(vals.cuda()), b.cuda(), x, rel_tol=rel_tol, abs_tol=1e-14)
        assert info["converged"] == 1 and info["found_indefiniteness"] == 0
        r = b.double().numpy() - A @ x.double().cpu().numpy()
        assert np.linalg.norm(r) <= 10 * rel_tol * np.linalg.norm(b.double().numpy())
