"""y = A x through symxg_bcsr_spmv_*: row counts around a thread block's 32 rows, empty rows, rows
longer than the 256 (in double 512) blocks that a thread block streams at a time, against float64.

Tolerance: a row of n terms is summed in some order, so |error| <= (n + 2) u sum |a| |x|, with u
the unit roundoff of the type (the float64 reference itself adds a few 2^-53 of the same sum)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("lengths", [[1], [0], [3] * 31, [15] * 32, [0, 16, 17, 0] * 8 + [5], [513, 0, 1, 1030] + [7] * 70,
                                     [0] * 40 + [2000]], ids=lambda v: f"{len(v)}rows_{sum(v)}")
def test_spmv_matches_float64(lib, dtype, lengths):
    import torch

    import symx_gb300 as sg

    rng = np.random.default_rng(len(lengths) + sum(lengths))
    n = len(lengths)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    cols = rng.integers(0, n, row_ptr[-1]).astype(np.int32)
    vals = rng.standard_normal((row_ptr[-1], 3, 3)).astype(dtype)
    x = rng.standard_normal(3 * n).astype(dtype)
    y = torch.full((3 * n,), 7.0, dtype=getattr(torch, dtype), device="cuda")
    dev = [torch.tensor(a, device="cuda") for a in (row_ptr, cols, vals, x)]
    if row_ptr[-1] == 0:  # torch's empty tensors have no address, which the entry point refuses
        with pytest.raises(sg.capi.SymxgError):
            sg.bcsr_spmv(dev[0], dev[1], sg.component_major(dev[2]), dev[3], y)
        return
    sg.bcsr_spmv(dev[0], dev[1], sg.component_major(dev[2]), dev[3], y)
    prod = vals.astype(np.float64) * x.astype(np.float64).reshape(-1, 1, 3)[cols]
    ref, size = np.zeros((n, 3)), np.zeros((n, 3))
    rows = np.repeat(np.arange(n), lengths)
    np.add.at(ref, rows, prod.sum(2))
    np.add.at(size, rows, np.abs(prod).sum(2))
    u = np.finfo(dtype).eps / 2
    bound = (3 * np.array(lengths)[:, None] + 2 + 8) * u * size
    assert np.all(np.abs(y.double().cpu().numpy().reshape(n, 3) - ref) <= bound)
