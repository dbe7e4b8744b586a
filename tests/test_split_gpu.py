"""GPU: the split variant of the any-dimension kernel (2D, 4D, 6D: half of the axes in registers, half
across the lanes) against the generic kernel, at element counts around the 32 / N^(D/2) elements of a
warp, with inflow on both sides, wrapped neighbours, a separate mass term and per-element factors."""
import numpy as np
import pytest
import torch

import gendil_b200 as g
from gendil_b200 import coefficients as C
from helpers import APPLY_TOL, cuda_apply, rel_max

pytestmark = pytest.mark.gpu

SHAPES = ([(2, p, s) for p in range(1, 8) for s in ([1, 1], [33, 2], [5, 7])] +
          [(4, p, s) for p in range(1, 5) for s in ([1, 1, 1, 1], [3, 2, 1, 2], [2, 3, 2, 3])] +
          [(6, p, s) for p in (1, 2) for s in ([1, 2, 1, 1, 1, 1], [2, 1, 3, 1, 2, 2])])


@pytest.mark.parametrize("D,p,sizes", SHAPES, ids=[f"{d}d_p{p}_{'x'.join(map(str, s))}" for d, p, s in SHAPES])
def test_split_variant_matches_generic(D, p, sizes):
    rng = np.random.default_rng(p)
    for periodic in (0, 1):
        sp = g.Space(D, sizes, [1.0 / n for n in sizes], None, [periodic] * D, p)
        factor = torch.from_numpy(rng.choice([-1.5, -0.5, 0.7, 1.3], sp.num_elements)).cuda()
        const = C.velocity_constant([0.7, -0.4, 0.25, -0.55, 0.3, -0.2][:D])
        for beta, sigma in ((C.velocity_bubble(D), C.Coefficient(terms=[{0: lambda x: 1 + x, D - 1: lambda x: 2 - x}])),
                            ([C.Coefficient(constant=c.constant, element_factor=factor) for c in const], 3.0)):
            op = g.SystemOperator(sp, p + 1, beta, sigma=sigma, g=0.3)
            assert op.kernel == "kronnd", op.kernel_note
            op.set_variant("nd-split")
            x = rng.uniform(-1, 1, sp.num_dofs)
            y, yt, y32 = cuda_apply(op, x), cuda_apply(op, x, transpose=True), cuda_apply(op, x, f32=True)
            try:
                op.select_kernel("generic")
            except g.DGOPError:
                op.set_variant("nd-passes")
            assert rel_max(y, cuda_apply(op, x)) <= APPLY_TOL
            assert rel_max(yt, cuda_apply(op, x, transpose=True)) <= APPLY_TOL
            assert rel_max(y32, y) <= 1e-5
