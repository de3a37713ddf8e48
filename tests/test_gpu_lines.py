"""Dispatch by size: both sides of each line, and the line itself.

Residual: one cell a CTA up to as many cells as CTAs are resident, two up to
twice as many, then four; against the oracle at the tolerances of
test_gpu_cells.  Sizes are those of a B200 (148 SMs); on another count they are
ordinary sizes."""
import pytest

import cpolyg_b200 as cp
import oracle
from cases import equations, rel, to_dev, to_np
from test_gpu_steppers import l2rel

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.mark.parametrize("name,deg,n", [("adv_rot", 1, 8 * SMS), ("adv_rot", 1, 8 * SMS + 1),
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
