"""The timed sweep form is decided once per class of preconditioners.  A class
holds preconditioners with the same candidates only: a matrix with a row too
long for the sync-free sweeps (more than 16 lower or upper blocks) has no
workspace for them, and stays with the level forms after another matrix of
its block size and number of rows has decided for a sync-free one.

The two-launch operator P^{-1} A is not what is timed there: every
preconditioner of a class takes it, whatever the class decided for its sweeps
and whether it was made before or after the decision."""
import numpy as np
import pytest
import torch

import cpolyg_b200 as cp
import oracle
from cases import mesh, rel, to_dev, to_np
from test_gpu_operator import fused

pytestmark = pytest.mark.gpu

SYNC_FREE = (1, 4, 5, 6)


def system(n, bl, hub):
    """A Voronoi pattern; hub > 0: row n - 1 is coupled to the first hub rows as well."""
    m, _, _ = mesh(n, True, 1.0, 2)
    rp, cl = m.pattern()
    rows = [list(cl[rp[i]:rp[i + 1]]) for i in range(n)]
    for j in range(hub):
        if n - 1 not in rows[j]:
            rows[j].append(n - 1)
            rows[n - 1].append(j)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    cl = np.concatenate(rows).astype(np.int32)
    rng = np.random.default_rng(bl + hub)
    blocks = rng.standard_normal((len(cl), bl, bl))
    for i in range(n):
        blocks[rp[i]] += np.eye(bl) * (3.0 * bl)
    return rp, cl, blocks


@pytest.mark.parametrize("bl", [6, 10, 24, 40])
@pytest.mark.parametrize("prec", [cp.F64, cp.F32])
def test_long_rows_do_not_take_another_matrix_form(ctx, bl, prec):
    n = 700
    form = cp.lib().cpg_precond_sweep_form
    short = cp.BlockILU0(cp.BlockMatrix.from_host(ctx, *system(n, bl, 0), precision=prec), precision=prec)
    x = np.random.default_rng(1).standard_normal(n * bl)
    short.solve(to_dev(x))  # decides its class
    assert form(short.h) != 0
    sysl = system(n, bl, 20)
    long = cp.BlockILU0(cp.BlockMatrix.from_host(ctx, *sysl, precision=prec), precision=prec)
    assert form(long.h) not in SYNC_FREE
    want = oracle.precond_apply(2, *sysl, x)
    # FP32 factors: 24 bits, and the factors' growth (cond of order 10)
    assert rel(to_np(long.solve(to_dev(x))), want) < (1e-11 if prec == cp.F64 else 1e-4)
    assert form(long.h) in (2, 3)


@pytest.mark.parametrize("form", [2, 3, 4, 5])
def test_operator_does_not_depend_on_the_decided_form(ctx, form):
    """Two preconditioners of one matrix, one created before its class decided
    for `form` and one after: the same operator, bit for bit, in one product
    and in a solve."""
    bl, n = 24, 900
    A = cp.BlockMatrix.from_host(ctx, *system(n, bl, 0))
    lib = cp.lib()
    assert lib.cpg_debug_decide_sweep_form(cp.BlockILU0(A).h, 0) == 0  # whatever came before
    before = cp.BlockILU0(A)
    assert lib.cpg_precond_sweep_form(before.h) == 0
    assert lib.cpg_debug_decide_sweep_form(before.h, form) == 0
    try:
        after = cp.BlockILU0(A)
        assert lib.cpg_precond_sweep_form(after.h) == form
        x = to_dev(np.random.default_rng(2).standard_normal(n * bl))
        y, z = fused(before, A, x), fused(after, A, x)
        assert torch.equal(y, z)
        assert not torch.equal(z, after.apply_op(A, x))  # it is the operator, not the product and the sweeps
        u, v = torch.zeros_like(x), torch.zeros_like(x)
        assert A.gmres(x, u, 20, 1e-10, 200, before) == A.gmres(x, v, 20, 1e-10, 200, after)
        assert torch.equal(u, v)
    finally:
        assert lib.cpg_debug_decide_sweep_form(before.h, 0) == 0
