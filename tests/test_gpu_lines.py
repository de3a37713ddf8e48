"""Dispatch by size: both sides of each line, and the line itself.

Sweeps: rows are polled up to so many rows a resident CTA (19 for form 4, 60
with 40x40 blocks) and go by flags from there on.  Both kernels sum as the
level form 2 does, so form 4 equals it bit for bit at any size.  Residual: one
cell a CTA (two at p = 1) up to as many cells as CTAs are resident, two up to
twice as many, then four; against the oracle at the tolerances of test_gpu_cells.  Sizes are
those of a B200 (148 SMs); on another count they are ordinary sizes."""
import numpy as np
import pytest
import torch

import cpolyg_b200 as cp
import oracle
from cases import equations, rel, to_dev, to_np
from test_gpu_operator import fused
from test_gpu_split import newton_system
from test_gpu_steppers import l2rel
from test_gpu_sweeps import bsr

pytestmark = pytest.mark.gpu

SMS = 148
LINE = {6: 19 * 10 * SMS, 10: 19 * 6 * SMS, 24: 19 * 5 * SMS, 40: 60 * 6 * SMS}
SYSTEM = {6: ("advection", 2), 10: ("advection", 3), 24: ("euler", 2), 40: ("euler", 3)}


def preconditioner(A, monkeypatch, form):
    monkeypatch.setenv("CPG_ILU_SWEEP", f"form{form}")
    P = cp.BlockILU0(A, precision=A.precision)
    monkeypatch.delenv("CPG_ILU_SWEEP")
    assert cp.lib().cpg_precond_sweep_form(P.h) == form
    return P


@pytest.mark.parametrize("bl", [6, 10, 24, 40])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_sweeps_at_the_line_between_polls_and_flags(ctx, monkeypatch, bl, off):
    if bl == 40 and off != 0:
        pytest.skip("4.8 GB a matrix: one side of the line is enough")
    n = LINE[bl] + off
    eq, u, _, J = newton_system(ctx, *SYSTEM[bl], n=n)
    P4, P2 = preconditioner(J, monkeypatch, 4), preconditioner(J, monkeypatch, 2)
    x = torch.randn(n * bl, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(7))
    want = P2.solve(x.clone())
    # the operator keeps its own state in the workspace that the sweeps use
    y = fused(P4, J, x)
    for _ in range(2):
        assert torch.equal(P4.solve(x.clone()), want)
        assert torch.equal(fused(P4, J, x), y)
    if bl == 40:
        return
    J32 = eq.jacobian(u, 0.0, scale=-1e-3, add_mass=True, precision=cp.F32)
    Q4, Q2 = preconditioner(J32, monkeypatch, 4), preconditioner(J32, monkeypatch, 2)
    assert torch.equal(Q4.solve(x.clone()), Q2.solve(x.clone()))


# rows of more threads: other lines, and sums in another order than form 2's
@pytest.mark.parametrize("bl,form,prec,line", [(6, 5, cp.F64, 16 * 5 * SMS), (10, 6, cp.F64, 16 * SMS),
                                               (24, 5, cp.F64, 25 * 2 * SMS), (40, 6, cp.F64, 25 * SMS),
                                               (10, 6, cp.F32, 24 * SMS), (24, 6, cp.F32, 47 * 3 * SMS)])
def test_wide_sweeps_at_their_lines(ctx, monkeypatch, bl, form, prec, line):
    for n in (line - 1, line):
        rp, cl, blocks = bsr(n, bl, bl)
        A = cp.BlockMatrix.from_host(ctx, rp, cl, blocks, precision=prec)
        del blocks
        Pw, P2 = preconditioner(A, monkeypatch, form), preconditioner(A, monkeypatch, 2)
        x = to_dev(np.random.default_rng(3).standard_normal(n * bl))
        y = Pw.solve(x.clone())
        assert rel(to_np(y), to_np(P2.solve(x.clone()))) < (1e-13 if prec == cp.F64 else 1e-6)
        assert torch.equal(Pw.solve(x.clone()), y)


@pytest.mark.parametrize("bl,n", [(6, 50001), (10, 50000)])
def test_sweeps_by_flags_match_oracle(ctx, monkeypatch, bl, n):
    rp, cl, blocks = bsr(n, bl, 11)
    P = preconditioner(cp.BlockMatrix.from_host(ctx, rp, cl, blocks), monkeypatch, 4)
    x = np.random.default_rng(5).standard_normal(n * bl)
    assert rel(to_np(P.solve(to_dev(x))), oracle.precond_apply(2, rp, cl, blocks, x)) < 1e-11


@pytest.mark.parametrize("name,deg,n", [("adv_rot", 1, 701), ("adv_rot", 1, 16 * SMS + 1),
                                        ("adv_rot", 3, 16 * SMS), ("adv_rot", 3, 16 * SMS + 1),
                                        ("euler", 1, 6 * SMS + 1), ("euler", 1, 12 * SMS + 1),
                                        ("euler", 2, 6 * SMS), ("euler", 2, 6 * SMS + 1),
                                        ("euler", 2, 12 * SMS), ("euler", 2, 12 * SMS + 3)])
def test_residual_at_its_lines(ctx, name, deg, n):
    ge, oe, _ = equations(ctx, name, deg, n=n, periodic=False)
    kind, params = (cp.INIT_VORTEX, [5.0, 0.5, 0.5, 1, 1, 1.4, 1, 1]) if name == "euler" else \
        (cp.INIT_GAUSSIAN, [30.0, 0.4, 0.6])
    u = oe.interp(kind, params)
    ug = to_dev(u).reshape(ge.np, ge.nc, ge.nb)
    assert rel(to_np(ge.assemble(ug, 0.1)), oe.assemble(u, 0.1)) < 1e-12
    x = ug.clone()
    cp.TimeStepper(ge, kind=cp.STEP_RK4).advance(x, 1e-4, 0.1)
    assert l2rel(to_np(x), oracle.Stepper(oe, cp.STEP_RK4).advance(u.copy(), 1e-4, 0.1)) < 1e-11
