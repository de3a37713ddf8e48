"""The two-launch operator P^{-1} A (A's lower blocks shared between the product
and the forward sweep) against the oracle's BlockILU0 and against the product
followed by the sweeps.

It regroups the sums of the lower blocks, A_ji D_i^{-1} y_i as A_ji (D_i^{-1}
y_i), so the two forms differ by the rounding of the stored L_ji, at most
about eps * cond(D_i) relative: 0.25 eps max cond_inf(D_i), the bound the
split form is held to, and 1e-11 against the oracle where cond is of order 10.
An accuracy between the split form's rounding and its own selects it."""
import numpy as np
import pytest
import torch

import cpolyg_b200 as cp
import oracle
from cases import mesh, rel, to_dev, to_np
from test_gpu_split import EPS, newton_system, rhs

pytestmark = pytest.mark.gpu


def fused(P, A, x):
    return P.apply_op(A, x, accuracy=0.1 * EPS * P.pivot_cond())


# 60 rows: a CTA each; 20,000: several rows a CTA at every block size
@pytest.mark.parametrize("bl", [6, 10, 24, 40])
@pytest.mark.parametrize("n,periodic", [(60, True), (61, False), (2500, True), (20000, True)])
def test_fused_operator_matches_oracle(ctx, bl, n, periodic):
    if n * bl > 500000 and bl > 10:
        n = 5000  # the oracle's share of the time
    m, _, _ = mesh(n, periodic, 1.0, 2)
    rp, cl = m.pattern()
    rng = np.random.default_rng(bl + n)
    blocks = rng.standard_normal((len(cl), bl, bl))
    for i in range(n):
        blocks[rp[i]] += np.eye(bl) * (3.0 * bl)
    A = cp.BlockMatrix.from_host(ctx, rp, cl, blocks)
    P = cp.BlockILU0(A)
    x = rng.standard_normal(n * bl)
    xd = to_dev(x)
    y = fused(P, A, xd)
    want = oracle.precond_apply(2, rp, cl, blocks, oracle.bsr_matvec(rp, cl, blocks, x))
    assert rel(to_np(y), want) < 1e-11
    # the workspace is left as the next application needs it
    assert torch.equal(fused(P, A, xd), y)


@pytest.mark.parametrize("physics,degree", [("advection", 2), ("advection", 3), ("euler", 2), ("euler", 3)])
def test_fused_operator_follows_the_matrix(ctx, physics, degree):
    eq, u, dt, J = newton_system(ctx, physics, degree)
    P = cp.BlockILU0(J)
    b = rhs(J)
    two_step = P.apply_op(J, b)
    y = fused(P, J, b)
    assert not torch.equal(y, two_step)
    assert rel(to_np(y), to_np(two_step)) < 0.25 * EPS * P.pivot_cond()
    # values that the factors are not those of: the product, then the sweeps
    eq.jacobian(u, 0.0, scale=-2 * dt * 0.435866521508459, add_mass=True, out=J)
    stale = P.apply_op(J, b)
    assert torch.equal(fused(P, J, b), stale) and not torch.equal(stale, two_step)
    P.refactor(J)
    again = fused(P, J, b)
    assert rel(to_np(again), to_np(P.apply_op(J, b))) < 0.25 * EPS * P.pivot_cond()
