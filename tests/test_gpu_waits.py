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


def test_a_solve_whose_wait_ran_out_ends_with_its_cycle(ctx):
    """The status word is read with every restart cycle.  A solve that finds it
    set reports the timeout then, instead of after all the cycles it may take."""
    lib = cp.lib()
    rp, cl, blocks = bsr(300, 6, 3)
    A = cp.BlockMatrix.from_host(ctx, rp, cl, blocks)
    P = cp.BlockILU0(A)
    b = to_dev(np.random.default_rng(0).standard_normal((len(rp) - 1) * 6))
    P.solve(b.clone())  # decides the sweep form
    m = 4
    before = ctx.launches
    A.gmres(b, torch.zeros_like(b), m, 1e-2, m, P)
    cycle = ctx.launches - before
    ctx.check(lib.cpg_ctx_set_deferred_checks(ctx.h, 1))
    try:
        assert lib.cpg_debug_wait_timeout(ctx.h, 1) == 0  # leaves the status word set
    finally:
        ctx.check(lib.cpg_ctx_set_deferred_checks(ctx.h, 0))
    before = ctx.launches
    with pytest.raises(cp.CpgError) as e:
        A.gmres(b, torch.zeros_like(b), m, 1e-15, 1000 * m, P)
    assert e.value.status == TIMEOUT
    assert ctx.launches - before < 2 * cycle
    its, res = A.gmres(b, torch.zeros_like(b), m, 1e-10, 1000 * m, P)
    assert res < 1e-10
