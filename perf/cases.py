"""The work a user of this framework has it do: operator applies, batches, gradients and solves, each
through the package's public entry points, over the sizes, orders, dimensions and types in use.

``listed()`` names the cases that are timed, ``draw(rng)`` gives more of the same ranges,
``prepare`` / ``run`` are a user's program, ``work`` / ``tolerance`` / ``exact`` say what a pass has
to move and compute, how far another correct implementation may be off, and what the result is (a
plain torch evaluation of the DG forms at the quadrature points in 64 bits, which shares nothing with
the package).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import gendil_b200 as g
from gendil_b200 import coefficients as C


def _case(kind, sizes, p, q, coef, name=None, basis="gll", dtype="f64", transpose=False):
    c = {"kind": kind, "D": len(sizes), "sizes": "x".join(str(n) for n in sizes), "p": p, "q": q, "coef": coef,
         "basis": basis, "dtype": dtype, "transpose": transpose}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # the smallest call: one mass apply on the CG test problem (262,144 DoFs, vectors in L2), where
        # launch and host cost count
        _case("mass", [16] * 3, 3, 4, "one", "mass_small"),
        # the benchmark's operator: upwind advection in a sheared velocity field, vectors larger than L2
        _case("advection", [64] * 3, 3, 4, "sincos", "advection"),
        # the adjoint direction on a mesh whose extents are no multiple of anything
        _case("advection", [37, 26, 31], 3, 4, "sincos", "advection_adjoint_ragged", transpose=True),
        # an implicit-Euler system operator M/dt + A at a higher order, over-integrated, ragged
        _case("system", [24, 19, 22], 5, 7, "sincos", "system_p5"),
        # the inner operator of the mixed-precision solvers
        _case("advection", [48] * 3, 3, 4, "sincos", "advection_f32", dtype="f32"),
        # 6D phase-space transport, 191 million DoFs: the largest state a user runs on one GPU
        _case("advection", [8] * 6, 2, 3, "phase", "advection_6d"),
        # a variable density that is no single product (the reference's own test field)
        _case("mass", [32] * 3, 3, 5, "poly", "mass_density"),
        # the Gauss-Legendre basis, the other basis of the reference, with a velocity along its own axis
        _case("advection", [32, 30, 33], 3, 4, "bubble", "advection_gauss", basis="gl"),
        # many independent small and middle systems applied together (2D to 4D, orders 1 to 5)
        {"name": "batch", "kind": "batch", "count": 24, "pick": 7, "emin": 1000, "emax": 20000},
        # interior-penalty diffusion and its coefficient gradient, one step of a coefficient fit
        _case("sipdg", [32] * 3, 4, 6, "lognormal", "diffusion_and_gradient"),
        # a diffusion solve by CG: hundreds of iterations of small kernels
        _case("cg", [12, 10, 11], 3, 5, "lognormal", "diffusion_cg"),
        # the implicit-Euler step of the benchmark: mixed-precision GMRES with the mass inverse
        _case("gmres", [64] * 3, 3, 4, "sincos", "implicit_step"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, D, elements):
    """D extents around the D-th root, whose product is about `elements`."""
    sizes, rest = [], float(elements)
    for k in range(D):
        n = rest ** (1.0 / (D - k)) * (rng.uniform(0.7, 1.4) if k < D - 1 else 1.0)
        sizes.append(max(1, int(round(n))))
        rest = max(1.0, rest / sizes[-1])
    rng.shuffle(sizes)
    return sizes


def draw(rng):
    kind = rng.choice(["mass", "advection", "advection", "advection", "system", "system", "phase", "batch", "sipdg",
                       "cg", "gmres"])
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 32), "pick": rng.randint(1, 10 ** 6), "emin": 500,
                "emax": _log_int(rng, 4000, 30000)}
    if kind == "phase":
        D = rng.choice([4, 6])
        sizes = [rng.choice([4, 6, 8]) if D == 6 else 2 * rng.randint(2, 12) for _ in range(D)]
        if D == 6 and math.prod(sizes) > 8 ** 6:
            sizes = [6] * 6
        p = rng.choice([1, 2]) if D == 6 else rng.randint(1, 4)
        return _case("advection", sizes, p, p + 1, "phase", dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "sipdg":
        p = rng.randint(1, 5)
        return _case("sipdg", _extents(rng, 3, _log_int(rng, 400, 4_000_000 / (p + 1) ** 3)), p, p + rng.randint(1, 2),
                     "lognormal")
    if kind == "cg":
        p = rng.randint(2, 4)
        return _case("cg", _extents(rng, 3, _log_int(rng, 200, 120_000 / (p + 1) ** 3 + 400)), p, p + 2, "lognormal")
    if kind == "gmres":
        p = rng.randint(2, 4)
        return _case("gmres", _extents(rng, 3, _log_int(rng, 4000, 17_000_000 / (p + 1) ** 3)), p, p + 1, "sincos")
    D = rng.choice([2, 3, 3, 3])
    p = rng.randint(1, 7 if D == 2 else 6)
    dofs = _log_int(rng, 200_000, 30_000_000)
    sizes = _extents(rng, D, dofs / (p + 1) ** D)
    if kind == "mass":
        coef = rng.choice(["one", "poly"])
    else:
        coef = rng.choice(["sincos", "sincos", "constant", "bubble"])
    basis = "gl" if rng.random() < 0.25 else "gll"
    return _case(kind, sizes, p, p + rng.randint(1, 2), coef, basis=basis,
                 dtype=rng.choice(["f64", "f64", "f64", "f32"]), transpose=kind == "advection" and rng.random() < 0.3)


# ------------------------------------------------------------------------------ a user's program

DT = 1e-3         # time step of the implicit-Euler systems
CG_TOL = 1e-10    # relative residual of the diffusion solves
GMRES_TOL = 1e-10


def _sizes(case):
    return [int(s) for s in case["sizes"].split("x")]


def _mesh(case):
    """(extents, h, origin): the unit cube, or [0, 1]^H x [-1, 1]^H for the phase-space field."""
    n = _sizes(case)
    H = len(n) // 2
    if case["coef"] == "phase":
        return n, [(1.0 if k < H else 2.0) / v for k, v in enumerate(n)], [0.0] * H + [-1.0] * H
    return n, [1.0 / v for v in n], [0.0] * len(n)


def _space(case):
    n, h, o = _mesh(case)
    return g.Space(len(n), n, h, o, None, case["p"], g.GL if case["basis"] == "gl" else g.GLL)


CONSTANT = (0.7, -0.4, 0.25, -0.55)


def _velocity(case):
    D = case["D"]
    if case["coef"] == "sincos":
        return C.velocity_sincos(D)
    if case["coef"] == "bubble":
        return C.velocity_bubble(D)
    if case["coef"] == "phase":
        return C.velocity_phase_space(D)
    return C.velocity_constant(CONSTANT[:D])


def _instances(case):
    """The systems of a batch: dimension 2 to 4, order 1 to 5, log-uniform element counts, constant
    velocities; drawn from the case, not from the inputs' seed."""
    rng = random.Random(case["pick"])
    out = []
    for _ in range(case["count"]):
        D, p = rng.randint(2, 4), rng.randint(1, 5)
        sizes = _extents(rng, D, _log_int(rng, case["emin"], case["emax"]))
        out.append({"D": D, "p": p, "n": sizes, "beta": [rng.uniform(-1.0, 1.0) for _ in range(D)]})
    return out


def _uniform(n, gen, dtype=torch.float64):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).mul_(2.0).sub_(1.0).to(dtype)


def _inputs(case, seed):
    """The vectors and the diffusivity of a case, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + int(seed))
    if case["kind"] == "batch":
        return {"xs": [_uniform(math.prod(d["n"]) * (d["p"] + 1) ** d["D"], gen) for d in _instances(case)]}
    n, ne = math.prod(_sizes(case)) * (case["p"] + 1) ** case["D"], math.prod(_sizes(case))
    v = {"x": _uniform(n, gen, torch.float32 if case["dtype"] == "f32" else torch.float64)}
    if case["coef"] == "lognormal":
        v["mu"] = torch.exp(0.5 * torch.randn(ne, dtype=torch.float64, device="cuda", generator=gen))
        if case["kind"] == "sipdg":
            v["lam"] = _uniform(n, gen)
    return v


def _kappa(case):
    return 10.0 * (case["p"] + 1) ** 2


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, **_inputs(case, seed)}
    if kind == "batch":
        ops = []
        for d in _instances(case):
            sp = g.Space(d["D"], d["n"], order=d["p"])
            ops.append(g.SystemOperator(sp, d["p"] + 2, C.velocity_constant(d["beta"]), sigma=1.0 / DT))
        s["ops"], s["batch"] = ops, g.Batch(ops)
        s["ys"] = [torch.empty_like(x) for x in s["xs"]]
        return s
    space = _space(case)
    q = case["q"]
    s["y"] = torch.empty_like(s["x"])
    if kind == "mass":
        s["op"] = g.MassOperator(space, q, 1.0 if case["coef"] == "one" else C.density_poly(case["D"]))
    elif kind == "advection":
        s["op"] = g.AdvectionOperator(space, q, _velocity(case), bc=g.BC_INFLOW, g=0.0)
    elif kind in ("system", "gmres"):
        s["op"] = g.SystemOperator(space, q, _velocity(case), sigma=1.0 / DT, bc=g.BC_INFLOW, g=0.0)
    else:
        s["op"] = g.SIPDGOperator(space, q, s["mu"], sigma=-1.0, kappa=_kappa(case), boundary=True)
    if kind == "sipdg":
        s["grad"] = torch.empty(space.num_elements, dtype=torch.float64, device="cuda")
    if kind == "cg":
        s["solver"] = g.CGSolver(s["op"])
    if kind == "gmres":
        s["prec"] = g.MassInverseOperator(space, q, 1.0 / DT)
        s["solver"] = g.GMRESIRSolver(s["op"], 30, inner="fp32").precondition(s["prec"])
    s["space"] = space
    s["apply"] = "f32" if case["dtype"] == "f32" else "transpose" if case["transpose"] else "plain"
    if case["dtype"] == "f32" and case["transpose"]:
        s["apply"] = "f32"  # the FP32 entry point has no transposed form
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].apply(s["xs"], s["ys"])
        return s["ys"]
    if kind == "sipdg":
        s["op"](s["x"], s["y"])
        s["op"].coefficient_gradient(s["x"], s["lam"], out=s["grad"])
        return {"y": s["y"], "grad": s["grad"]}
    if kind in ("cg", "gmres"):
        s["y"].zero_()
        s["solver"].solve(s["x"], s["y"], 20000, CG_TOL if kind == "cg" else GMRES_TOL)
        return s["y"]
    if s["apply"] == "f32":
        return s["op"].apply_f32(s["x"], s["y"])
    if s["apply"] == "transpose":
        return s["op"].apply_transpose(s["x"], s["y"])
    return s["op"](s["x"], s["y"])


# ------------------------------------------------------------------- what a pass cannot do without


def _apply_flops(kind, D, p, dofs):
    """Sum factorization along the axes, 2 (p + 1) flops per value and axis: one sweep for a mass
    term, one per axis for an advection or diffusion operator."""
    terms = {"mass": 1, "advection": D, "system": D + 1}.get(kind, D)
    return 2.0 * (p + 1) * D * terms * dofs


def work(case):
    """Inputs read once, outputs written once, in the vectors' type.  The solvers count the applies
    and the vector passes of an iteration for the iterations these systems take (about 50 per element
    along the longest axis and order in CG, about 50 in GMRES with the mass inverse)."""
    if case["kind"] == "batch":
        b = f = 0.0
        for d in _instances(case):
            n = math.prod(d["n"]) * (d["p"] + 1) ** d["D"]
            b += 16.0 * n
            f += _apply_flops("system", d["D"], d["p"], n)
        return {"bytes": b, "flops": f}
    sizes, D, p = _sizes(case), case["D"], case["p"]
    n = math.prod(sizes) * (p + 1) ** D
    size = 4 if case["dtype"] == "f32" else 8
    one = {"bytes": 2.0 * size * n, "flops": _apply_flops(case["kind"], D, p, n)}
    if case["kind"] == "sipdg":
        return {"bytes": 2 * one["bytes"] + 16.0 * math.prod(sizes), "flops": 3 * one["flops"]}
    if case["kind"] == "cg":
        its = 50.0 * max(sizes) * p
        return {"bytes": its * (one["bytes"] + 56.0 * n), "flops": its * (one["flops"] + 10.0 * n)}
    if case["kind"] == "gmres":
        # an iteration in 32 bits: the system and the mass apply, and half a restart's basis, twice
        return {"bytes": 50.0 * (16.0 * n + 2 * 15 * 4.0 * n), "flops": 50.0 * (2 * one["flops"] + 60.0 * n)}
    return one


def tolerance(case):
    """Four times what the path shows against exact(), rounded up: rounding of the vectors' type
    for an apply (up to 2.0e-15 in 64 bits, 9.3e-8 in 32); for a solve the residual it stops at, seen
    through the system's conditioning (2.4e-10 for CG, 6.4e-11 for GMRES)."""
    if case["kind"] == "cg":
        return {"rel": 2e-9}
    if case["kind"] == "gmres":
        return {"rel": 5e-10}
    if case["kind"] == "batch":
        return {"rel": 1e-14}
    return {"rel": 4e-7} if case["dtype"] == "f32" else {"rel": 1e-14}


# ------------------------------------------------------------- the same in plain torch, in 64 bits


def _gll(p):
    """The p + 1 Gauss-Lobatto-Legendre points on [0, 1]."""
    if p == 0:
        return np.array([0.5])
    inner = np.polynomial.legendre.Legendre.basis(p).deriv().roots().real
    for _ in range(4):  # Newton on P_p' with P_p'' from Legendre's equation
        L = np.polynomial.legendre.Legendre.basis(p)
        inner = inner - L.deriv()(inner) / L.deriv(2)(inner)
    return 0.5 * (1.0 + np.concatenate([[-1.0], np.sort(inner), [1.0]]))


def _lagrange(nodes, x):
    """(values, derivatives) of the Lagrange basis on `nodes` at the points x: len(x) x len(nodes)."""
    n = len(nodes)
    V, G = np.ones((len(x), n)), np.zeros((len(x), n))
    for i in range(n):
        for k in range(n):
            if k != i:
                V[:, i] *= (x - nodes[k]) / (nodes[i] - nodes[k])
        for m in range(n):
            if m != i:
                t = np.full(len(x), 1.0 / (nodes[i] - nodes[m]))
                for k in range(n):
                    if k not in (i, m):
                        t = t * (x - nodes[k]) / (nodes[i] - nodes[k])
                G[:, i] += t
    return V, G


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


class _Forms:
    """The DG forms on a Cartesian mesh: vectors as (n_{D-1}, .., n_0, N, .., N), axis 0 last."""

    def __init__(self, D, n, h, origin, p, q, gl=False):
        self.D, self.n, self.h, self.origin, self.N = D, n, h, origin, p + 1
        x, w = np.polynomial.legendre.leggauss(q)
        self.xq, self.w = 0.5 * (x + 1.0), 0.5 * w
        nodes = 0.5 * (np.polynomial.legendre.leggauss(p + 1)[0] + 1.0) if gl else _gll(p)
        B, G = _lagrange(nodes, self.xq)
        F, dF = _lagrange(nodes, np.array([0.0, 1.0]))
        self.M1 = B.T @ (self.w[:, None] * B)
        self.B, self.G, self.F, self.dF = _dev(B), _dev(G), _dev(F), _dev(dF)
        self.detJ = math.prod(h)

    def shape(self, x):
        return x.reshape(self.n[::-1] + [self.N] * self.D)

    def along(self, M, u, k):
        """M applied along the values' axis k."""
        d = 2 * self.D - 1 - k
        return torch.movedim(torch.movedim(u, d, -1) @ M.T, -1, d)

    def at_points(self, fn, k, face=None):
        """fn at the points (or on the face) along axis k, shaped to multiply a values array."""
        e = self.origin[k] + self.h[k] * np.arange(self.n[k])
        x = e[:, None] + self.h[k] * (self.xq[None, :] if face is None else np.array([[float(face)]]))
        s = [1] * (2 * self.D)
        s[self.D - 1 - k], s[2 * self.D - 1 - k] = x.shape
        return _dev(fn(x)).reshape(s)

    def coef(self, terms, a=None, face=None):
        """sum of products of functions of one coordinate, at the cell's points or a face's."""
        v = 0.0
        for t in terms:
            m = torch.ones([1] * (2 * self.D), dtype=torch.float64, device="cuda") * t.get("c", 1.0)
            for k, fn in t.items():
                if k != "c":
                    m = m * self.at_points(fn, k, face if k == a else None)
            v = v + m
        return v

    def weighted(self, u, skip=None):
        for k in range(self.D):
            if k != skip:
                s = [1] * (2 * self.D)
                s[2 * self.D - 1 - k] = len(self.w)
                u = u * _dev(self.w).reshape(s)
        return u * self.detJ

    def interp(self, u, skip=None):
        for k in range(self.D):
            if k != skip:
                u = self.along(self.B, u, k)
        return u

    def test(self, v, skip=None, grad=None):
        for k in range(self.D):
            if k != skip:
                v = self.along((self.G if k == grad else self.B).T, v, k)
        return v

    def neighbour(self, t, a, s):
        """The value on the neighbour across side s of axis a; zero outside the domain."""
        d = self.D - 1 - a
        r = torch.roll(t, -1 if s else 1, d)
        edge = [slice(None)] * t.dim()
        edge[d] = slice(self.n[a] - 1, self.n[a]) if s else slice(0, 1)
        keep = torch.ones([self.n[a] if i == d else 1 for i in range(t.dim())], dtype=torch.float64, device="cuda")
        keep[tuple(slice(None) if i != d else edge[d] for i in range(t.dim()))] = 0.0
        return r * keep, keep

    def mass(self, u, terms):
        return self.test(self.weighted(self.interp(u) * self.coef(terms)))

    def advection(self, u, beta):
        """-(u beta, grad v) + <upwind flux, v>, inflow value 0."""
        ui = self.interp(u)
        y = 0.0
        for a in range(self.D):
            y = y + self.test(self.weighted(-ui * (self.coef(beta[a]) / self.h[a])), grad=a)
        del ui
        for a in range(self.D):
            for s in (0, 1):
                own = self.interp(self.along(self.F[s:s + 1], u, a), skip=a)
                other, _ = self.neighbour(self.interp(self.along(self.F[1 - s:2 - s], u, a), skip=a), a, s)
                bn = self.coef(beta[a], a, s) * ((1.0 if s else -1.0) / self.h[a])
                flux = self.weighted(bn.clamp(min=0.0) * own + bn.clamp(max=0.0) * other, skip=a)
                y = y + self.along(self.F[s:s + 1].T, self.test(flux, skip=a), a)
        return y

    def sipdg(self, u, mu, sigma, kappa):
        """Interior penalty with one diffusivity per element, Dirichlet 0: cells, interior and boundary facets."""
        m = mu.reshape(self.n[::-1] + [1] * self.D)
        ui = self.interp(u)
        y = 0.0
        for a in range(self.D):
            du = u
            for k in range(self.D):
                du = self.along(self.G if k == a else self.B, du, k)
            y = y + self.test(self.weighted(m * du / self.h[a] ** 2), grad=a)
        del ui
        for a in range(self.D):
            for s in (0, 1):
                nu, hi = (1.0 if s else -1.0), 1.0 / self.h[a]
                face = lambda R, v: self.interp(self.along(R, v, a), skip=a)  # noqa: E731
                t, d = face(self.F[s:s + 1], u), face(self.dF[s:s + 1], u) * hi
                tn, keep = self.neighbour(face(self.F[1 - s:2 - s], u), a, s)
                dn, _ = self.neighbour(face(self.dF[1 - s:2 - s], u) * hi, a, s)
                mn, _ = self.neighbour(m, a, s)
                # inside: averages over the two sides; on the boundary the own value alone
                half = 1.0 - 0.5 * keep
                grad = nu * (half * m * d + 0.5 * mn * dn)
                mbar = half * m + 0.5 * mn
                jump = t - tn
                val = self.weighted((-grad + kappa * hi * mbar * jump) * hi, skip=a)
                der = self.weighted(sigma * jump * half * m * nu * hi * hi, skip=a)
                y = y + self.along(self.F[s:s + 1].T, self.test(val, skip=a), a)
                y = y + self.along(self.dF[s:s + 1].T, self.test(der, skip=a), a)
        return y


def _beta_terms(case):
    D, H = case["D"], case["D"] // 2
    two_pi = 2.0 * np.pi
    if case["coef"] == "constant":
        return [[{"c": CONSTANT[a]}] for a in range(D)]
    if case["coef"] == "bubble":
        return [[{a: lambda x: -x * (1.0 - x)}] for a in range(D)]
    if case["coef"] == "phase":
        return [[{a + H: lambda x: x}] if a < H else [{a - H: lambda x: 0.5 - x}] for a in range(D)]
    rows = [[{1 % D: lambda x: 1.0 + 0.5 * np.sin(two_pi * x)}], [{2 % D: lambda x: 0.5 + 0.25 * np.cos(two_pi * x)}]]
    return (rows + [[{"c": 0.25}] for _ in range(D)])[:D]


def _density_terms(case):
    if case["coef"] == "one":
        return [{}]
    D = case["D"]
    return [{}, {0: lambda x: x, 1: lambda x: x}, {D - 1: lambda x: x * x}]


def _gmres(apply, prec, b, tol, most=150):
    """Right-preconditioned full GMRES with two Gram-Schmidt passes."""
    V, H = [b / b.norm()], torch.zeros(most + 1, most, dtype=torch.float64)
    for j in range(most):
        w = apply(prec(V[j]))
        for _ in range(2):
            for i, v in enumerate(V):
                c = torch.dot(v, w)
                H[i, j] += c.item()
                w = w - c * v
        H[j + 1, j] = w.norm().item()
        V.append(w / H[j + 1, j])
        e = torch.zeros(j + 2, 1, dtype=torch.float64)
        e[0] = b.norm().item()
        y = torch.linalg.lstsq(H[:j + 2, :j + 1], e).solution
        if (H[:j + 2, :j + 1] @ y - e).norm().item() < tol * b.norm().item():
            break
    x = torch.zeros_like(b)
    for i in range(y.shape[0]):
        x += y[i, 0].item() * V[i]
    return prec(x)


def exact(case, seed):
    v = _inputs(case, seed)
    if case["kind"] == "batch":
        out = []
        for d, x in zip(_instances(case), v["xs"]):
            f = _Forms(d["D"], d["n"], [1.0 / n for n in d["n"]], [0.0] * d["D"], d["p"], d["p"] + 2)
            u = f.shape(x)
            out.append((f.mass(u, [{"c": 1.0 / DT}]) + f.advection(u, [[{"c": b}] for b in d["beta"]])).reshape(-1))
        return out
    n, h, o = _mesh(case)
    kind = case["kind"]
    f = _Forms(case["D"], n, h, o, case["p"], case["q"], case["basis"] == "gl")
    x = v["x"].double()
    flat = lambda fn: lambda t: fn(f.shape(t)).reshape(-1)  # noqa: E731
    if kind == "mass":
        return f.mass(f.shape(x), _density_terms(case)).reshape(-1)
    if kind in ("sipdg", "cg"):
        kappa = _kappa(case)
        if kind == "sipdg":
            y = f.sipdg(f.shape(x), v["mu"], -1.0, kappa).reshape(-1)
            mu = v["mu"].clone().requires_grad_(True)
            dot = (f.sipdg(f.shape(x), mu, -1.0, kappa).reshape(-1) * v["lam"]).sum()
            return {"y": y, "grad": torch.autograd.grad(dot, mu)[0]}
        A = flat(lambda u: f.sipdg(u, v["mu"], -1.0, kappa))
        u, r = torch.zeros_like(x), x.clone()
        d, rr = r.clone(), torch.dot(r, r)
        for _ in range(6000):
            ad = A(d)
            a = rr / torch.dot(d, ad)
            u, r = u + a * d, r - a * ad
            new = torch.dot(r, r)
            if new.item() < (1e-13 * x.norm().item()) ** 2:
                return u
            d, rr = r + (new / rr) * d, new
        return None
    beta = _beta_terms(case)
    if kind == "advection":
        if case["transpose"] and case["dtype"] == "f64":
            u = torch.zeros_like(x).requires_grad_(True)
            return torch.autograd.grad((f.advection(f.shape(u), beta).reshape(-1) * x).sum(), u)[0]
        return f.advection(f.shape(x), beta).reshape(-1)
    A = flat(lambda u: f.mass(u, [{"c": 1.0 / DT}]) + f.advection(u, beta))
    if kind == "system":
        return A(x)
    Minv = _dev(np.linalg.inv(f.M1))

    def prec(t):
        t = f.shape(t)
        for k in range(f.D):
            t = f.along(Minv, t, k)
        return (t * (DT / f.detJ)).reshape(-1)

    return _gmres(A, prec, x, 1e-13)
