"""The bounded waits of the one-launch PCG with the matrix in shared memory (k_pcg_resident) run out, in
any iteration: with a small limit on the polls some waits succeed and some give up, in some of the
blocks.  A call then fails with the error of a bounded wait or gives the bits of an unlimited one, in
bounded time (a wait that gives up ends every other wait of its block), and the next call is as
before.  Systems with a gather list, without one (random columns), and of a single block."""
import time

import numpy as np
import pytest

from test_gpu_pcg_resident import _spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,offsets,per_row", [(15, (1, 2), 0), (2433, (1, 40, 41, 1200), 0), (20000, (), 60)])
def test_waits_give_up_together(lib, n, offsets, per_row, dtype):
    import torch

    import symx_gb300 as sg

    rp, cols, vals = _spd(n, offsets, per_row, seed=n)
    t = getattr(torch, dtype)
    args = [torch.tensor(rp, device="cuda"), torch.tensor(cols, device="cuda"),
            sg.component_major(torch.tensor(vals, dtype=t, device="cuda")),
            torch.tensor(np.random.default_rng(n).standard_normal(3 * n), dtype=t, device="cuda")]
    x = torch.empty(3 * n, dtype=t, device="cuda")
    ref_info = sg.bcsr_pcg(*args, x)
    ref = x.clone()
    assert ref_info["converged"] == 1
    gave_up = 0
    try:
        for limit in (0, 1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 64, 256):
            lib.symxg_set_wait_poll_limit(limit)
            for _ in range(4):
                x.fill_(float("nan"))
                start = time.perf_counter()
                try:
                    info = sg.bcsr_pcg(*args, x)
                    assert limit > 0 and info == ref_info and torch.equal(x, ref)
                except sg.SymxgError as e:
                    assert "bounded wait" in str(e)
                    gave_up += 1
                assert time.perf_counter() - start < 5.0
    finally:
        lib.symxg_set_wait_poll_limit(-1)
    assert gave_up >= 4
    assert sg.bcsr_pcg(*args, x) == ref_info and torch.equal(x, ref)
