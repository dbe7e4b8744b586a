"""GPU: batches of independent operators (dgop_batch_apply): one persistent launch per
(dimension, order, kernel variant) group on the any-dimension Kronecker kernel, the rest one launch each; results
bit-identical to each operator's own apply."""
import numpy as np
import pytest
import torch

import gendil_b200 as g
from gendil_b200 import coefficients as C

pytestmark = pytest.mark.gpu


def _space(D, n, p, basis=g.GLL):
    sizes = n if isinstance(n, list) else [n] * D
    return g.Space(D, sizes, [1.0 / s for s in sizes], [0.0] * D, None, p, basis)


def _batched(o):
    """Whether the persistent batch kernel serves this operator's variant: every any-dimension
    variant but the mass-only one, with blocks of at most 27 values (N = order + 1; grouped by 2
    axes up to N = 5, by 3 up to N = 3, paired up to N = 5)."""
    if o.kernel != "kronnd":
        return False
    n = o.space.order + 1
    return {"nd-passes": True, "nd-grouped2": n * n <= 27, "nd-grouped3": n ** 3 <= 27,
            "nd-paired": n * n <= 27}.get(o.variant, False)


def test_batch_apply_equals_individual_applies():
    rng = np.random.default_rng(7)
    ops = []
    for D, n, p in [(2, [9, 7], 3), (2, [5, 11], 3), (3, [4, 3, 5], 4), (4, [3, 2, 4, 3], 1), (2, [6, 6], 1),
                    (3, [3, 3, 3], 4), (4, [2, 3, 2, 2], 2), (3, [5, 4, 3], 2), (2, [7, 5], 5)]:
        sp = _space(D, n, p)
        beta = C.velocity_constant(list(rng.uniform(-1, 1, D)))
        ops.append(g.SystemOperator(sp, p + 2, beta, sigma=1e3, bc=g.BC_INFLOW, g=0.0))
    ops.append(g.SystemOperator(_space(2, [4, 5], 2, g.GL), 4, C.velocity_constant([0.3, -0.7]), sigma=1e3))
    kinds = [o.kernel for o in ops]
    assert "kronnd" in kinds and "kron" in kinds and "generic" in kinds
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = []
    for o, x in zip(ops, xs):
        y = torch.empty_like(x)
        o(x, y)
        want.append(y)
    batch = g.Batch(ops)
    assert batch.groups == len({(o.space.dim, o.space.order, o.variant) for o in ops if _batched(o)})
    for _ in range(2):  # twice: the parameter upload of the previous apply is reused safely
        ys = [torch.full_like(x, float("nan")) for x in xs]
        batch.apply(xs, ys)
        torch.cuda.synchronize()
        for y, w in zip(ys, want):
            assert torch.equal(y, w)
    batch.close()


def test_batch_large_instance_keeps_its_own_launch():
    """An instance whose element batches fill every CTA slot of the GPU twice over (here 10^6
    elements) is applied by its own launch, outside the groups; the small instances of the same
    (dimension, order) still form a group, and every result is bit-identical to its own apply."""
    rng = np.random.default_rng(11)
    specs = [(2, [1000, 1000], 1), (2, [9, 7], 1), (2, [5, 11], 1)]
    ops = []
    for D, n, p in specs:
        beta = C.velocity_constant(list(rng.uniform(-1, 1, D)))
        ops.append(g.SystemOperator(_space(D, n, p), p + 2, beta, sigma=1e3, bc=g.BC_INFLOW, g=0.0))
    for o in ops[1:]:
        o.set_variant(ops[0].variant)  # one (dimension, order, variant) key for all three
    assert all(o.kernel == "kronnd" for o in ops)
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = []
    for o, x in zip(ops, xs):
        y = torch.empty_like(x)
        o(x, y)
        want.append(y)
    batch = g.Batch(ops)
    assert batch.groups == 1
    ys = [torch.full_like(x, float("nan")) for x in xs]
    batch.apply(xs, ys)
    torch.cuda.synchronize()
    for y, w in zip(ys, want):
        assert torch.equal(y, w)
    batch.close()


def test_batch_unbatched_variant_runs_one_launch_each():
    """Operators whose variant has no persistent batch kernel (2D p = 5 on 36-value blocks of 2
    axes) form no group and are applied one launch each, bit-identical to their own applies."""
    rng = np.random.default_rng(5)
    ops = []
    for n in ([7, 5], [6, 9]):
        beta = C.velocity_constant(list(rng.uniform(-1, 1, 2)))
        o = g.SystemOperator(_space(2, n, 5), 7, beta, sigma=1e3, bc=g.BC_INFLOW, g=0.0)
        o.set_variant("nd-grouped2")
        ops.append(o)
    assert not any(_batched(o) for o in ops)
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = []
    for o, x in zip(ops, xs):
        y = torch.empty_like(x)
        o(x, y)
        want.append(y)
    batch = g.Batch(ops)
    assert batch.groups == 0
    ys = [torch.full_like(x, float("nan")) for x in xs]
    batch.apply(xs, ys)
    torch.cuda.synchronize()
    for y, w in zip(ys, want):
        assert torch.equal(y, w)
    batch.close()


def _systems(specs, seed=7):
    rng = np.random.default_rng(seed)
    ops, precs, bs = [], [], []
    for D, n, p in specs:
        sp = _space(D, n, p)
        beta = C.velocity_constant(list(rng.uniform(-1, 1, D)))
        ops.append(g.SystemOperator(sp, p + 2, beta, sigma=1e3, bc=g.BC_INFLOW, g=0.0))
        precs.append(g.MassInverseOperator(sp, p + 2, 1e3))
        bs.append(torch.tensor(rng.uniform(-1, 1, sp.num_dofs), device="cuda"))
    return ops, precs, bs


SOLVE_SPECS = [(2, [40, 33], 3), (3, [12, 10, 9], 2), (4, [6, 5, 4, 5], 1), (3, [16, 8, 8], 3), (2, [25, 30], 5),
               (4, [4, 4, 3, 3], 3), (3, [7, 9, 8], 4)]


@pytest.mark.parametrize("inner", ["fp32", "fp64"])
def test_batch_solver_matches_single_system_solves(inner):
    """The lockstep batched refinement GMRES(20) reaches the same 1e-10 FP64 residual as the
    single-system solver on every system, in the same number of iterations within one (their
    inner products sum in different fixed orders), with solutions equal to rounding; the reported
    residual is the true one."""
    ops, precs, bs = _systems(SOLVE_SPECS)
    batch = g.BatchSolver(ops, precs, restart=20, inner=inner)
    xs = [torch.zeros_like(b) for b in bs]
    res, secs = batch.solve(bs, xs, 2000, 1e-10)
    for A, P, b, x, r, t in zip(ops, precs, bs, xs, res, secs):
        assert r["success"] and r["relative_error"] <= 1e-10, r
        ax = torch.empty_like(x)
        A(x, ax)
        true_rel = (torch.linalg.vector_norm(b - ax) / torch.linalg.vector_norm(b)).item()
        assert abs(true_rel - r["relative_error"]) <= 1e-3 * r["relative_error"] + 1e-15
        x1 = torch.zeros_like(b)
        one = g.GMRESIRSolver(A, 20, inner=inner).precondition(P).solve(b, x1, 2000, 1e-10)
        assert abs(one["iterations"] - r["iterations"]) <= 1, (one, r)
        assert ((x - x1).abs().max() / x1.abs().max()).item() <= 1e-8
        assert t > 0.0


def test_batch_solver_waves_are_independent():
    """Cutting the systems into several waves (a small workspace budget) changes nothing: every
    system's computation depends on its own vectors and partial sums only (bit-identical)."""
    ops, precs, bs = _systems(SOLVE_SPECS, seed=9)
    one = g.BatchSolver(ops, precs, restart=20, inner="fp32")
    many = g.BatchSolver(ops, precs, restart=20, inner="fp32", workspace_bytes=8e6)
    assert one.waves == 1 and many.waves >= 3
    xa = [torch.zeros_like(b) for b in bs]
    xb = [torch.zeros_like(b) for b in bs]
    ra, _ = one.solve(bs, xa, 2000, 1e-10)
    rb, _ = many.solve(bs, xb, 2000, 1e-10)
    assert ra == rb
    for a, b in zip(xa, xb):
        assert torch.equal(a, b)
    # a second solve from the found solutions: the true residual is already below tol
    rc, _ = one.solve(bs, xa, 2000, 1e-10)
    assert all(r["success"] and r["iterations"] == 0 for r in rc)


def test_batch_solver_reports_unconverged_systems():
    ops, precs, bs = _systems(SOLVE_SPECS[:3], seed=11)
    batch = g.BatchSolver(ops, precs, restart=5, inner="fp32")
    xs = [torch.zeros_like(b) for b in bs]
    res, _ = batch.solve(bs, xs, 3, 1e-14)
    assert all(not r["success"] and r["iterations"] == 3 and r["relative_error"] > 1e-14 for r in res)


def _passes_ops(count, rng):
    """`count` operators of one group whose batch kernel runs for hundreds of microseconds (one
    shared-memory pass per axis, 110,592 DoFs each)."""
    ops = []
    for _ in range(count):
        o = g.SystemOperator(_space(3, 12, 3), 5, C.velocity_constant(list(rng.uniform(-1, 1, 3))), sigma=1e3)
        o.select_kernel("kronnd")
        o.set_variant("nd-passes")
        ops.append(o)
    return ops


def test_batch_on_two_streams_without_a_wait():
    """Applies of one batch on two unordered streams, different vectors each: the second apply's
    parameter table must not replace the first one's under its kernels."""
    rng = np.random.default_rng(3)
    ops = _passes_ops(24, rng)
    ops += [g.SystemOperator(_space(2, [9, 7], 3), 5, C.velocity_constant([0.3, -0.4]), sigma=1e3) for _ in range(3)]
    batch = g.Batch(ops)
    assert batch.groups >= 1
    streams = [torch.cuda.Stream() for _ in range(2)]
    xs = [[torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops] for _ in streams]
    want = [[o(x, torch.empty_like(x)) for o, x in zip(ops, v)] for v in xs]
    for _ in range(10):
        ys = [[torch.full_like(x, float("nan")) for x in v] for v in xs]
        torch.cuda.synchronize()
        for s, x, y in zip(streams, xs, ys):
            batch.apply(x, y, stream=s)
        torch.cuda.synchronize()
        for w, y in zip(want, ys):
            assert all(torch.equal(a, b) for a, b in zip(w, y))
    batch.close()


def test_batch_applied_by_two_threads():
    """Two host threads apply one batch, each on a stream of its own."""
    import threading
    rng = np.random.default_rng(4)
    ops = _passes_ops(4, rng) + [g.SystemOperator(_space(3, n, 3), 5, C.velocity_constant([0.5, -0.2, 0.1]), sigma=1e3)
                                 for n in ([5, 4, 3], [8, 3, 2], [7, 7, 7])]
    batch = g.Batch(ops)
    xs = [[torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops] for _ in range(2)]
    want = [[o(x, torch.empty_like(x)) for o, x in zip(ops, v)] for v in xs]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                ys = [torch.full_like(x, float("nan")) for x in xs[k]]
                batch.apply(xs[k], ys, stream=s)
                s.synchronize()
                if not all(torch.equal(a, b) for a, b in zip(want[k], ys)):
                    wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    batch.close()


def test_batch_with_a_repeated_operator_that_owns_a_workspace():
    """Several right-hand sides of one operator in a batch, whose element (729 values, 4^6 points) does
    not fit in shared memory: the generic kernel then works in one global workspace per operator,
    which the members' applies must use in turn.  Another operator's launches run beside them."""
    sp = _space(6, [2, 3, 2, 2, 2, 2], 2, g.GL)
    rng = np.random.default_rng(6)
    op = g.SystemOperator(sp, 4, C.velocity_constant(list(rng.uniform(-1, 1, 6))), sigma=1e3)
    assert op.kernel == "generic"
    other = g.SystemOperator(_space(3, [5, 4, 3], 3), 5, C.velocity_constant([0.5, -0.2, 0.1]), sigma=1e3)
    ops = [op, other, op, op, other, op, op, op]
    batch = g.Batch(ops)
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = [o(x, torch.empty_like(x)) for o, x in zip(ops, xs)]
    for _ in range(5):
        ys = [torch.full_like(x, float("nan")) for x in xs]
        batch.apply(xs, ys)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, ys))
    batch.close()


@pytest.mark.parametrize("D,p,count,n", [(2, 1, 60, 60), (2, 2, 12, 60), (2, 5, 6, 40), (2, 7, 4, 20), (4, 1, 6, 6),
                                         (4, 3, 4, 4), (6, 1, 4, 3), (6, 2, 4, 2)])
def test_split_variant_groups(D, p, count, n):
    """Groups of the split variant, with more element batches than the batch kernel has CTAs for the small
    orders (a CTA moves from one instance to the next and takes its matrices), extents that differ
    from instance to instance, and velocities that vary along an axis in every other one."""
    rng = np.random.default_rng(D * 10 + p)
    ops = []
    for i in range(count):
        sp = _space(D, [n + i % 3] + [n] * (D - 1), p)
        beta = C.velocity_sincos(D) if i % 2 else C.velocity_constant(list(rng.uniform(-1, 1, D)))
        o = g.SystemOperator(sp, min(8, p + 2), beta, sigma=1e3)
        o.set_variant("nd-split")
        ops.append(o)
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = [o(x, torch.empty_like(x)) for o, x in zip(ops, xs)]
    batch = g.Batch(ops)
    assert batch.groups == 1
    ys = [torch.full_like(x, float("nan")) for x in xs]
    batch.apply(xs, ys)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, ys))
    batch.close()


@pytest.mark.parametrize("inner", ["fp32", "fp64"])
def test_batch_solver_with_a_repeated_operator_that_owns_a_workspace(inner):
    """Several right-hand sides of one operator whose applies share a global workspace (see the batched
    apply's test), beside another system: every system as when solved by itself (cut off after 40
    steps, with the residual reached by then)."""
    op = g.SystemOperator(_space(6, [2, 1, 2, 2, 1, 2], 2, g.GL), 4, C.velocity_constant([0.3, -0.2, 0.5, 0.1, -0.4, 0.2]),
                          sigma=1e3)
    assert op.kernel == "generic"
    other = g.SystemOperator(_space(3, [5, 4, 3], 3), 5, C.velocity_constant([0.5, -0.2, 0.1]), sigma=1e3)
    ops = [op, other, op, op, op]
    bs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    xs = [torch.zeros_like(b) for b in bs]
    res, _ = g.BatchSolver(ops, None, restart=10, inner=inner).solve(bs, xs, 40, 1e-10)
    for o, b, x, r in zip(ops, bs, xs, res):
        alone = torch.zeros_like(b)
        (one,), _ = g.BatchSolver([o], None, restart=10, inner=inner).solve([b], [alone], 40, 1e-10)
        assert one == r and torch.equal(alone, x)


@pytest.mark.parametrize("specs", [[(3, 5, 3), (3, 6, 2), (3, 4, 4)],
                                   [(2, 9, 1), (2, 11, 1), (4, 4, 2), (4, 3, 2), (4, 5, 2), (4, 3, 2), (3, 4, 3)]],
                         ids=["single_launches", "groups"])
def test_batch_under_stream_capture(specs):
    """A captured batched apply replays with the vectors it was captured with, whatever the batch did
    in between, and the batch applies eagerly before and after."""
    rng = np.random.default_rng(8)
    ops = []
    for D, n, p in specs:
        o = g.SystemOperator(_space(D, n, p), p + 2, C.velocity_constant(list(rng.uniform(-1, 1, D))), sigma=1e3)
        if D % 2 == 0:
            o.set_variant("nd-split")
        ops.append(o)
    batch = g.Batch(ops)
    assert batch.groups == (2 if len(specs) > 3 else 0)
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    ys, other = [torch.zeros_like(x) for x in xs], [torch.zeros_like(x) for x in xs]
    batch.apply(xs, other)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        batch.apply(xs, ys)
    for _ in range(2):
        for x in xs:
            x.mul_(-0.5)
        want = [o(x, torch.empty_like(x)) for o, x in zip(ops, xs)]
        batch.apply([w.clone() for w in want], other)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want))


@pytest.mark.parametrize("p", [4, 5])
def test_small_3d_operators_above_order_3_share_launches(p):
    """More operators than one launch takes, of both term structures, from one element to several CTAs,
    velocities constant and varying, periodic and not: bit for bit their own applies, also with one vector
    off 16 bytes (whose launch falls back to single applies)."""
    rng = np.random.default_rng(p)
    ops = []
    for i in range(24):
        sizes = [1 + i % 5, 1 + i % 3, 1 + i % 4] if i else [9, 8, 7]
        sp = g.Space(3, sizes, [1.0 / n for n in sizes], None, [i % 2, 0, (i // 2) % 2], p)
        beta = C.velocity_sincos(3) if i % 4 == 1 else C.velocity_constant(list(rng.uniform(-1, 1, 3)))
        sigma = C.Coefficient(terms=[{0: lambda x: 1 + x}]) if i >= 12 else 1e3
        ops.append(g.SystemOperator(sp, p + 2, beta, sigma=sigma, bc=g.BC_INFLOW, g=0.3))
        assert ops[-1].kernel == "kron", ops[-1].kernel_note
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    want = [o(x, torch.empty_like(x)) for o, x in zip(ops, xs)]
    batch = g.Batch(ops)
    assert 2 <= batch.groups <= 6
    for off in (None, 3):
        ys = [torch.full_like(x, float("nan")) for x in xs]
        if off is not None:
            ys[off] = torch.full((xs[off].numel() + 1,), float("nan"), dtype=torch.float64, device="cuda")[1:]
        batch.apply(xs, ys)
        torch.cuda.synchronize()
        for k, (y, w) in enumerate(zip(ys, want)):
            if k == off:  # the any-dimension kernel
                assert float((y - w).abs().max()) <= 1e-13 * float(w.abs().max())
            else:
                assert torch.equal(y, w), k
    batch.close()


def test_batch_follows_a_kernel_chosen_after_it_was_made():
    """Operators of a group, and of a shared launch, whose kernel is chosen anew after the batch was made are
    applied as their own applies are."""
    ops = [g.SystemOperator(_space(2, n, 2), 4, C.velocity_constant([0.3, -0.4]), sigma=1e3) for n in (9, 11, 7, 8)]
    for o in ops:
        o.set_variant("nd-split")
    ops += [g.SystemOperator(_space(3, n, 4), 6, C.velocity_constant([0.3, -0.4, 0.2]), sigma=1e3) for n in (3, 4, 2, 3)]
    xs = [torch.rand(o.space.num_dofs, dtype=torch.float64, device="cuda") - 0.5 for o in ops]
    batch = g.Batch(ops)
    assert batch.groups == 2
    for change in (None, 0, 4):
        if change is not None:
            ops[change].select_kernel("generic")
        want = [o(x, torch.empty_like(x)) for o, x in zip(ops, xs)]
        ys = [torch.full_like(x, float("nan")) for x in xs]
        batch.apply(xs, ys)
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want)), change
