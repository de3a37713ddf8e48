"""GMRES over the exponent range.  The basis is kept before normalisation, yet
a solve must take every right-hand side whose norm is representable.  Scaling
the matrix by 2^a and the right-hand side by 2^c scales every quantity of the
iteration by a power of two and the solution by 2^(c-a), so the solution of the
scaled system is that of the plain one scaled, bit for bit.  With a = c = 400
a dot product of two vectors that both carry |b| would be of order 2^1200."""
import numpy as np
import pytest
import torch

import cpolyg_b200 as cp
from cases import to_dev
from test_gpu_sweeps import bsr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,c", [(400, 400), (-400, -400), (0, 480), (0, -480), (300, -300), (-300, 300)])
@pytest.mark.parametrize("pc,flexible", [(None, False), (cp.BlockJacobi, True), (cp.BlockILU0, True),
                                         (cp.BlockILU0, False)])
def test_scaled_systems_have_scaled_solutions(ctx, a, c, pc, flexible):
    if pc is cp.BlockILU0 and not flexible and abs(c - a) > 500:
        pytest.skip("P^{-1} b is of order 2^(c-a): its norm is formed from squares, which have to be representable")
    bl, n = 6, 400
    rp, cl, blocks = bsr(n, bl, 9)
    b = np.random.default_rng(4).standard_normal(n * bl)
    x = {}
    for k, (sa, sb) in enumerate(((0, 0), (a, c))):
        A = cp.BlockMatrix.from_host(ctx, rp, cl, np.ldexp(blocks, sa))
        P = pc(A) if pc else None
        x[k] = torch.zeros(n * bl, dtype=torch.float64, device="cuda")
        its, res = A.gmres(to_dev(np.ldexp(b, sb)), x[k], 30, 1e-9, 300, P, flexible=flexible)
        x[k, "its"] = (its, res)
        assert res < 1e-9
    assert x[0, "its"] == x[1, "its"]
    assert torch.equal(x[0] * 2.0 ** (c - a), x[1])
