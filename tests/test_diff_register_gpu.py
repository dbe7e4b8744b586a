"""GPU: the 3D register kernel of the diffusion operator (16-byte aligned vectors) against the
shared-memory kernel (other vectors): apply, alpha / beta, FP32, element ranges, the fused inner product
of CG and the coefficient gradient."""
import numpy as np
import pytest
import torch

import gendil_b200 as g
from helpers import rel_max

pytestmark = pytest.mark.gpu

# orders 1..5; element counts around a warp's group of 32 / (p + 1); one-element and two-element
# periodic axes (a neighbour that is the element itself, or on both sides)
SHAPES = [(p, s, per, basis) for p in range(1, 6) for s, per, basis in
          (([32 // (p + 1) + 1, 2, 3], [0, 0, 0], g.GLL), ([1, 2, 3], [1, 1, 0], g.GLL), ([5, 4, 1], [0, 1, 1], g.GL))]


def _offset(t):
    """The same values at an address that is 8 bytes off a 16-byte boundary."""
    base = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    base[1:].copy_(t)
    return base[1:]


@pytest.mark.parametrize("p,sizes,periodic,basis", SHAPES)
@pytest.mark.parametrize("sigma,boundary", [(-1.0, True), (1.0, False)])
def test_register_kernel_matches_shared_memory_kernel(p, sizes, periodic, basis, sigma, boundary):
    sp = g.Space(3, sizes, [0.3, 0.2, 0.5], None, periodic, p, basis)
    gen = torch.Generator(device="cuda").manual_seed(p)
    rand = lambda n: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5  # noqa: E731
    mu = torch.exp(rand(sp.num_elements))
    op = g.SIPDGOperator(sp, p + 1, mu, sigma=sigma, boundary=boundary)
    x, lam, y0 = rand(sp.num_dofs), rand(sp.num_dofs), rand(sp.num_dofs)
    y, want = torch.empty_like(x), _offset(x)
    op(x, y)
    op(_offset(x), want)
    scale = float(want.abs().max())
    assert float((y - want).abs().max()) <= 1e-13 * scale
    yb = y0.clone()
    op.apply(x, yb, alpha=1.5, beta=-0.25)
    assert float((yb - (1.5 * y - 0.25 * y0)).abs().max()) <= 1e-14 * max(scale, 1.0)
    z = torch.empty(sp.num_dofs, dtype=torch.float32, device="cuda")
    op.apply_f32(x.float(), z)
    assert float((z.double() - want).abs().max()) <= 1e-5 * scale
    grad, gwant = op.coefficient_gradient(x, lam, scale=mu), op.coefficient_gradient(_offset(x), lam, scale=mu)
    # the sums of a gradient entry: 1e-13 of the largest product they contain
    assert float((grad - gwant).abs().max()) <= 1e-13 * max(float(gwant.abs().max()), scale)
    io = g.HostIO(op, slabs=2)
    xh = x.cpu()
    yh = torch.empty_like(xh)
    io.apply(xh, yh)
    assert torch.equal(yh, y.cpu())
    io.close()


def test_cg_with_fused_product_matches_separate_pass():
    sp = g.Space(3, [5, 4, 3], order=3)
    mu = torch.exp(0.3 * torch.randn(sp.num_elements, dtype=torch.float64, device="cuda",
                                     generator=torch.Generator(device="cuda").manual_seed(1)))
    op = g.SIPDGOperator(sp, 5, mu)
    b = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, sp.num_dofs)).cuda()
    got = []
    for fused in (True, True, False):
        x = torch.zeros_like(b)
        info = g.CGSolver(op).fused_dot(fused).solve(b, x, 5000, 1e-10)
        assert info["success"]
        got.append((x, info))
    assert torch.equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
    # the same products in another fixed order: iterates agree to the stopping tolerance
    assert rel_max(got[0][0].cpu().numpy(), got[2][0].cpu().numpy()) <= 1e-8


@pytest.mark.parametrize("p", range(1, 6))
def test_gauss_legendre_with_a_wrapped_x_axis(p):
    """Wrapped x neighbours, which are not in the staged group, on a basis whose traces are whole lines: the
    apply and the coefficient gradient, FP32, and CG with the fused inner product (p = 5 has none on a mesh
    this small: its apply is the shared-memory kernel's)."""
    sp = g.Space(3, [32 // (p + 1) + 2, 2, 3], [0.3, 0.2, 0.5], None, [1, 0, 0], p, g.GL)
    gen = torch.Generator(device="cuda").manual_seed(p)
    rand = lambda n: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5  # noqa: E731
    mu = torch.exp(rand(sp.num_elements))
    op = g.SIPDGOperator(sp, p + 1, mu)
    x, lam = rand(sp.num_dofs), rand(sp.num_dofs)
    y, want = op(x, torch.empty_like(x)), op(_offset(x), _offset(x))
    scale = float(want.abs().max())
    assert float((y - want).abs().max()) <= 1e-13 * scale
    z = op.apply_f32(x.float(), torch.empty(sp.num_dofs, dtype=torch.float32, device="cuda"))
    assert float((z.double() - want).abs().max()) <= 1e-5 * scale
    grad, gwant = op.coefficient_gradient(x, lam), op.coefficient_gradient(_offset(x), lam)
    assert float((grad - gwant).abs().max()) <= 1e-13 * max(float(gwant.abs().max()), scale)
    got = []
    for fused in (True, False):
        u = torch.zeros_like(x)
        assert g.CGSolver(op).fused_dot(fused).solve(x, u, 5000, 1e-10)["success"]
        got.append(u)
    # the same products in another fixed order: iterates agree to the stopping tolerance
    assert rel_max(got[0].cpu().numpy(), got[1].cpu().numpy()) <= 1e-8


@pytest.mark.parametrize("elements", [12 * 13 * 13, 13 * 13 * 13])
def test_order_5_apply_on_either_side_of_the_small_mesh_limit(elements):
    """Below 2048 elements the FP64 apply at p = 5 is the shared-memory kernel's, bit for bit that of vectors off
    16 bytes; above, the register kernel's, which sums in another order."""
    sizes = [elements // 169, 13, 13]
    sp = g.Space(3, sizes, order=5)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda n: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5  # noqa: E731
    op = g.SIPDGOperator(sp, 6, torch.exp(rand(sp.num_elements)))
    x = rand(sp.num_dofs)
    y, off = op(x, torch.empty_like(x)), op(_offset(x), _offset(x))
    assert torch.equal(y, off) == (elements < 2048)
    assert float((y - off).abs().max()) <= 1e-13 * float(off.abs().max())
