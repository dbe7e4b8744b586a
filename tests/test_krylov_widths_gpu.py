"""GPU: the basis kernels of the restarted solvers at every width of a projection pass (compiled per
number of vectors up to 16, further rows of 16) and with dofs that do not fill a 16-byte access: the
returned solution has the residual that the stopping test asks for."""
import pytest
import torch

import gendil_b200 as g
from gendil_b200 import coefficients as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1, 2, 15, 16, 17, 33])
@pytest.mark.parametrize("inner", ["gmres", "fp64", "fp32"])
def test_restarts_around_a_pass(inner, restart):
    tol = 1e-8
    for n in (37, 38, 39, 40):  # 3 n dofs: every remainder modulo 4
        sp = g.Space(1, [n], order=2)
        # sigma well above the transport rate beta (2 p + 1) / h of the coarsest mesh, so that short
        # restarts converge too, in more steps than the longest one
        op = g.SystemOperator(sp, 4, C.velocity_constant([1.0]), sigma=1e3)
        gen = torch.Generator(device="cuda").manual_seed(n)
        b = torch.rand(sp.num_dofs, dtype=torch.float64, device="cuda", generator=gen) - 0.5
        x = torch.zeros_like(b)
        s = g.GMRESSolver(op, restart) if inner == "gmres" else g.GMRESIRSolver(op, restart, inner=inner)
        info = s.solve(b, x, 4000, tol)
        assert info["success"], (n, info)
        r = b - op(x, torch.empty_like(x))
        # the estimate of the last step against the true residual: rounding of a few hundred steps
        assert r.norm() <= (tol + 1e-12) * b.norm() * (1 + 1e-4)
