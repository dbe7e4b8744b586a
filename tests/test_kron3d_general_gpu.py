"""GPU: the 3D register kernel over the orders and forms it takes (p = 0..5, bases without nodes on
the faces, densities that are sums of products, per-element factors), against the oracle or the
generic kernel."""
import math

import numpy as np
import pytest
import torch

import gendil_b200 as g
from gendil_b200 import coefficients as C
from helpers import APPLY_TOL, cuda_apply, inputs, make_operator, oracle, rel_max

pytestmark = pytest.mark.gpu


def _case(p, q, sizes, basis=0, beta=2, sigma=0, periodic=(0, 0, 0), gval=0.5, c=None):
    return {"D": 3, "P": p, "Q": q, "basis": basis, "sizes": list(sizes), "h": [1.0 / n for n in sizes],
            "origin": [0.0] * 3, "periodic": list(periodic), "beta_kind": beta, "beta_c": c, "sigma_kind": sigma,
            "sigma_c": 2.0, "g": gval, "seed": 3}


# element counts around the warp's group (32 / (p + 1) elements), inflow on either or both sides of
# an axis, wrapped neighbours inside and outside the group, varying and constant matrices
CASES = ([("p%d" % p, _case(p, p + 2, (7, 3, 5))) for p in range(6)] +
         [("p%d_bubble" % p, _case(p, p + 1, (32 // (p + 1) + 1, 2, 3), beta=1)) for p in (1, 4, 5)] +
         [("p%d_wrap" % p, _case(p, p + 1, (5, 4, 3), beta=0, c=[-0.7, 0.4, -0.3], periodic=(1, 1, 1)))
          for p in (2, 4, 5)] +
         [("gl%d" % p, _case(p, p + 1, (6, 5, 4), basis=1, beta=b)) for p, b in ((0, 0), (1, 1), (2, 2), (3, 1), (4, 1), (5, 2))] +
         [("gl3_wrap", _case(3, 5, (9, 3, 2), basis=1, beta=0, c=[0.6, -0.2, 0.5], periodic=(1, 0, 1)))] +
         [("poly%d" % p, _case(p, p + 1, (6, 3, 7), sigma=1)) for p in (1, 3, 4, 5)] +
         [("gl2_poly", _case(2, 4, (5, 4, 3), basis=1, beta=1, sigma=1))])
for _, _c in CASES:
    if _c["beta_kind"] == 0 and _c["beta_c"] is None:
        _c["beta_c"] = [0.7, -0.4, 0.25]


@pytest.mark.parametrize("case", [c for _, c in CASES], ids=[n for n, _ in CASES])
def test_register_kernel_matches_oracle_and_generic(case):
    x = inputs(case)
    for kind, mode in (("mass", 1), ("adv", 0), ("adv", 1), ("adv", 2)):
        op = make_operator(case, kind, mode)
        assert op.kernel == "kron", op.kernel_note
        want = oracle().mass_apply(case, x) if kind == "mass" else oracle().advection_apply(case, x, mode)
        y = cuda_apply(op, x)
        assert rel_max(y, want) <= APPLY_TOL, (kind, mode)
        yt, y32 = cuda_apply(op, x, transpose=True), cuda_apply(op, x, f32=True)
        xd = torch.from_numpy(x).cuda()
        yb = torch.from_numpy(x[::-1].copy()).cuda()
        op.apply(xd, yb, alpha=2.5, beta=-0.5)
        assert rel_max(yb.cpu().numpy(), 2.5 * y - 0.5 * x[::-1]) <= 1e-14
        try:
            op.select_kernel("generic")
        except g.DGOPError:
            continue  # no generic kernel for this shape
        assert rel_max(yt, cuda_apply(op, x, transpose=True)) <= APPLY_TOL, (kind, mode)
        # FP32: each of the three contractions rounds sums of N (N + 1) / 2-term products; 1e-5 of
        # the largest value as for the other FP32 applies
        assert rel_max(y32, y) <= 1e-5, (kind, mode)


@pytest.mark.parametrize("basis", [g.GLL, g.GL])
@pytest.mark.parametrize("p", [2, 3, 5])
def test_per_element_factors_are_read_at_every_apply(p, basis):
    """Velocity factors changed in place (signs included) between applies: the upwind decisions
    follow the new values, as on the generic kernel."""
    sp = g.Space(3, [8, 3, 4], order=p, basis=basis)
    rng = np.random.default_rng(1)
    factor = torch.from_numpy(rng.uniform(0.5, 1.5, sp.num_elements)).cuda()
    beta = [C.Coefficient(constant=v, element_factor=factor) for v in (0.8, -0.5, 0.3)]
    op = g.SystemOperator(sp, p + 1, beta, sigma=C.Coefficient(constant=3.0, element_factor=factor))
    gen = g.SystemOperator(sp, p + 1, beta, sigma=C.Coefficient(constant=3.0, element_factor=factor))
    assert op.kernel == "kron", op.kernel_note
    gen.select_kernel("generic")
    x = rng.uniform(-1, 1, sp.num_dofs)
    for _ in range(2):
        for tr in (False, True):
            assert rel_max(cuda_apply(op, x, transpose=tr), cuda_apply(gen, x, transpose=tr)) <= APPLY_TOL
        factor.mul_(torch.from_numpy(rng.choice([-1.0, 1.0], sp.num_elements)).cuda())


def test_sums_that_are_one_product_are_merged():
    """A constant plus functions of one coordinate is one separable product: such velocities and
    densities take the Kronecker kernels in every dimension, with the generic kernel's results."""
    for D, sizes in ((2, [5, 7]), (3, [5, 4, 3])):
        sp = g.Space(D, sizes, order=3)
        beta = [C.Coefficient(constant=1.0, terms=[{(a + 1) % D: lambda x: 0.5 * x * x}, {(a + 1) % D: lambda x: 0.2 * x}])
                for a in range(D)]
        op = g.SystemOperator(sp, 5, beta, sigma=C.Coefficient(constant=2.0, terms=[{0: lambda x: x}]))
        assert op.kernel == ("kronnd" if D == 2 else "kron"), op.kernel_note
        x = np.random.default_rng(0).uniform(-1, 1, sp.num_dofs)
        y = cuda_apply(op, x)
        op.select_kernel("generic")
        assert rel_max(y, cuda_apply(op, x)) <= APPLY_TOL


def test_mass_inverse_stays_limited_to_single_products():
    sp = g.Space(3, [3, 3, 3], order=2)
    with pytest.raises(g.DGOPError):
        g.MassInverseOperator(sp, 4, C.Coefficient(constant=1.0, terms=[{0: lambda x: x}]))
    with pytest.raises(g.DGOPError):
        g.MassInverseOperator(g.Space(3, [3, 3, 3], order=2, basis=g.GL), 4, 1.0)


@pytest.mark.parametrize("p", [4, 5])
def test_vectors_off_16_bytes_above_order_3(p):
    """Vectors aligned to their element size only, and operators without a generic kernel among them,
    run on the any-dimension kernel above order 3."""
    sp = g.Space(3, [4, 3, 5], order=p)
    rng = np.random.default_rng(p)
    x = torch.from_numpy(rng.uniform(-1, 1, sp.num_dofs)).cuda()
    off = torch.empty(sp.num_dofs + 1, dtype=torch.float64, device="cuda")
    out = torch.empty_like(off)
    off[1:] = x
    for op in (g.SystemOperator(sp, p + 2, C.velocity_sincos(3), sigma=2.0), g.MassInverseOperator(sp, p + 2, 2.0)):
        assert op.kernel == "kron", op.kernel_note
        y = op(x, torch.empty_like(x))
        for xs, ys in ((off[1:], out[1:]), (x, out[1:]), (off[1:], torch.empty_like(x))):
            assert rel_max(op(xs, ys).cpu().numpy(), y.cpu().numpy()) <= APPLY_TOL


def test_each_form_is_tuned_on_its_own():
    """Operators that differ by the kernel they run (basis, per-element factors, which matrices vary), but not
    in order, quadrature, flags and size, get their own timings whatever was created before them."""
    sizes = [9, 7, 5]
    factor = torch.full((math.prod(sizes),), 0.5, dtype=torch.float64, device="cuda")
    beta = C.velocity_constant([0.7, -0.4, 0.25])
    ops = [g.AdvectionOperator(g.Space(3, sizes, order=3), 4, beta),
           g.AdvectionOperator(g.Space(3, sizes, order=3, basis=g.GL), 4, beta),
           g.AdvectionOperator(g.Space(3, sizes, order=3), 4, C.velocity_bubble(3)),
           g.AdvectionOperator(g.Space(3, sizes, order=3), 4,
                               [C.Coefficient(constant=c.constant, element_factor=factor) for c in beta])]
    times = [tuple(sorted(op.variant_times().items())) for op in ops]
    assert all(op.kernel == "kron" for op in ops) and len(set(times)) == len(ops)
    again = g.AdvectionOperator(g.Space(3, sizes, order=3), 4, beta)  # the same form: the record of the first
    assert tuple(sorted(again.variant_times().items())) == times[0]


@pytest.mark.parametrize("p", [4, 5])
def test_any_dimension_kernel_of_register_operators_is_tuned(p):
    """Above order 3, where vectors off 16 bytes run on the any-dimension kernel, its variants are timed at
    creation as for the operators that always run there."""
    sp = g.Space(3, [6, 5, 4], order=p)
    for op in (g.SystemOperator(sp, p + 2, C.velocity_sincos(3), sigma=2.0), g.MassOperator(sp, p + 2, 2.0)):
        assert op.kernel == "kron", op.kernel_note
        op.select_kernel("kronnd")
        times = {k: t for k, t in op.variant_times().items() if t > 0.0}
        assert len(times) >= 2 and times[op.variant] == min(times.values())


@pytest.mark.parametrize("D,p,kernel", [(1, 1, "generic"), (1, 4, "generic"), (2, 1, "kronnd"), (2, 5, "kronnd"),
                                        (2, 6, "generic"), (3, 3, "kron"), (3, 6, "kronnd"), (4, 1, "kronnd")])
def test_gauss_legendre_mass_takes_the_faster_kernel(D, p, kernel):
    """The any-dimension kernel where it has its mass-only variant, and in 3D; the generic kernel, as for
    every basis without face nodes, elsewhere.  Same values on either."""
    sp = g.Space(D, [5, 3, 4, 2][:D], order=p, basis=g.GL)
    op = g.MassOperator(sp, p + 1, 1.5)
    assert op.kernel == kernel, op.kernel_note
    x = np.random.default_rng(D + p).uniform(-1, 1, sp.num_dofs)
    y, y32 = cuda_apply(op, x), cuda_apply(op, x, f32=True)
    op.select_kernel("generic")
    assert rel_max(y, cuda_apply(op, x)) <= APPLY_TOL and rel_max(y32, y) <= 1e-5


@pytest.mark.parametrize("p", range(1, 6))
def test_fp32_rounding_of_the_register_kernel(p):
    """The FP32 apply's error (2-norm, against the FP64 apply) is that of the any-dimension kernel, which
    contracts axis by axis and adds whole terms: the same roundings in another order, which move a norm
    over 10^4 values and more by a few per cent.  (Terms summed onto one another's partial sums, at
    the size of all of them, take 6 to 21 % more.)"""
    sp = g.Space(3, [11, 10, 9], order=p)
    op = g.AdvectionOperator(sp, p + 1, C.velocity_sincos(3))
    assert op.kernel == "kron", op.kernel_note
    x = np.random.default_rng(p).uniform(-1, 1, sp.num_dofs).astype(np.float32).astype(np.float64)
    y = cuda_apply(op, x)
    err = []
    for kernel in ("kron", "kronnd"):
        op.select_kernel(kernel)
        err.append(np.linalg.norm(cuda_apply(op, x, f32=True) - y))
    assert err[0] <= 1.05 * err[1], err


@pytest.mark.parametrize("basis", [g.GLL, g.GL])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
def test_system_with_a_density_that_is_a_sum(p, basis):
    """Advection terms and the mass terms of a sum of products in one launch, with a per-element density
    factor: forward, transposed and FP32, against the generic kernel."""
    sp = g.Space(3, [32 // (p + 1) + 1, 2, 3], order=p, basis=basis)
    factor = torch.from_numpy(np.random.default_rng(p).uniform(0.5, 1.5, sp.num_elements)).cuda()
    density = C.density_poly(3)
    sigma = C.Coefficient(constant=density.constant, terms=density.terms, element_factor=factor)
    op = g.SystemOperator(sp, p + 2, C.velocity_sincos(3), sigma=sigma, bc=g.BC_INFLOW, g=0.3)
    assert op.kernel == "kron", op.kernel_note
    x = np.random.default_rng(p + 1).uniform(-1, 1, sp.num_dofs)
    y, yt, y32 = cuda_apply(op, x), cuda_apply(op, x, transpose=True), cuda_apply(op, x, f32=True)
    op.select_kernel("generic")
    assert rel_max(y, cuda_apply(op, x)) <= APPLY_TOL and rel_max(yt, cuda_apply(op, x, transpose=True)) <= APPLY_TOL
    assert rel_max(y32, y) <= 1e-5
