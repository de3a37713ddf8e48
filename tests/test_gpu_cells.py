"""The residual's cells per CTA (one, two or four, by the mesh's size) and the
stage block Jacobi's block widths, against the oracle.

Sizes lie on either side of the lines at five and ten cells an SM (148 SMs),
with a remainder in the last CTA.  Tolerances are those the same kernels are
held to elsewhere: 1e-12 for a residual, which sums the same quadrature terms
in another order, and 1e-11 for a step."""
import pytest

import cpolyg_b200 as cp
import oracle
from cases import equations, rel, to_dev, to_np
from test_gpu_steppers import GAUSS, l2rel, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 740, 741, 1479, 1480, 1481, 1485])
@pytest.mark.parametrize("name,deg,periodic", [("adv_rot", 1, False), ("euler", 2, False), ("euler", 3, True)])
def test_residual_and_rk_stages_at_every_cta_size(ctx, name, deg, periodic, n):
    if n < 20 and periodic:
        pytest.skip("a periodic mesh needs more cells")
    ge, oe, _ = equations(ctx, name, deg, n=n, periodic=periodic)
    kind, params = (cp.INIT_VORTEX, [5.0, 0.5, 0.5, 1, 1, 1.4, 1, 1]) if name == "euler" else \
        (cp.INIT_GAUSSIAN, [30.0, 0.4, 0.6])
    u = oe.interp(kind, params)
    ug = to_dev(u).reshape(ge.np, ge.nc, ge.nb)
    assert rel(to_np(ge.assemble(ug, 0.1)), oe.assemble(u, 0.1)) < 1e-12
    for kind in (cp.STEP_FORWARD_EULER, cp.STEP_RK2, cp.STEP_RK4):
        x = ug.clone()
        cp.TimeStepper(ge, kind=kind).advance(x, 1e-4, 0.1)
        assert l2rel(to_np(x), oracle.Stepper(oe, kind).advance(u.copy(), 1e-4, 0.1)) < 1e-11


# stage blocks of 9 (no pairs), 12, 18 and 30 rows
@pytest.mark.parametrize("kind,deg", [(cp.STEP_IRK3, 1), (cp.STEP_IRK2, 2), (cp.STEP_IRK3, 2), (cp.STEP_IRK3, 3)])
def test_stage_block_jacobi_widths(ctx, kind, deg):
    ug, uo, gs, _ = run_both(ctx, "adv_const", deg, kind, 150, 1.0, 1, 0.005, pc=cp.PC_STAGE_BJACOBI, gm=40,
                             gtol=1e-13, gmaxit=20000, init=GAUSS, oracle_pc=3)
    assert gs.stats.converged == 1
    assert l2rel(ug, uo) < 1e-11
