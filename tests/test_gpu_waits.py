"""Bounded waits of the kernels whose rows wait for other rows.

Each kernel is run on a row whose dependency is never published: its wait runs
out, the call reports CPG_ERR_TIMEOUT, the status word is cleared, and the
context and its preconditioners work as before."""
import numpy as np
import pytest
import torch

import cpolyg_b200 as cp
import oracle
from cases import rel, to_dev, to_np
from test_gpu_operator import fused
from test_gpu_sweeps import bsr

pytestmark = pytest.mark.gpu

TIMEOUT = 6  # CPG_ERR_TIMEOUT
KERNELS = ["ring", "polled", "flags", "op_forward", "op_backward", "split_forward", "split_backward"]


@pytest.mark.parametrize("kernel", range(7), ids=KERNELS)
def test_wait_runs_out_and_is_reported(ctx, kernel):
    lib = cp.lib()
    rp, cl, blocks = bsr(300, 6, 3)
    A = cp.BlockMatrix.from_host(ctx, rp, cl, blocks)
    P = cp.BlockILU0(A)
    x = np.random.default_rng(0).standard_normal((len(rp) - 1) * 6)
    before = fused(P, A, to_dev(x))
    assert lib.cpg_debug_wait_timeout(ctx.h, kernel) == TIMEOUT, lib.cpg_last_error(ctx.h)
    assert rel(to_np(P.solve(to_dev(x))), oracle.precond_apply(2, rp, cl, blocks, x)) < 1e-11
    assert torch.equal(fused(P, A, to_dev(x)), before)
    assert lib.cpg_debug_wait_timeout(ctx.h, 7) != 0 and lib.cpg_debug_wait_timeout(ctx.h, -1) != 0
    ctx.sync()  # nothing left to report
