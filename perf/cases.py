"""The calls a user of this framework makes, as timed cases.

    listed()            named cases: solves, single cycles, assemblies, gradients
    draw(rng)           one more case of the same kinds and size ranges
    prepare(case, seed) a context with its levels set up and the call's inputs
    run(state)          one call through gascoignelib_b200.native.Context
    work(case)          bytes and operations the call cannot do without
    exact(case, seed)   the call's result in 64 bits, by plain torch

Kinds. "solve": one linear solve from host vector to host vector, the call that
replaces the reference's NewtonLinearSolve; the fields smoother, method and
mgtype are the solver keys. "cycle": one multigrid cycle as the preconditioner
of a Krylov loop that runs on the host. "newton": the matrices of all levels
from a new coefficient field, and the Newton residual. "design": one step of a
design loop, i.e. assembly, forward solve, functional, adjoint solve and the
gradient with respect to the coefficients.

A size is `coarse` and `refine`: coarse * 2^refine cells per dimension (ball:
refined once more inside a ball, with hanging nodes), `refine` levels.
"""
import dataclasses
import functools

import numpy as np
import torch

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import (kappa_pyramid, q2_meshes, stokes_rhs, structured_meshes,
                                       structured_problem, structured_q2, structured_q2_ball,
                                       structured_stokes)

LEFT, FLEXIBLE64, MIXED = 0, 1, 2  # method of gb_solve_host
BETA = (1.0, 0.5, 0.25)            # convection of the Q2 problems
EPS = 1e-2


def listed():
    def case(name, kind, disc, dim, coarse, refine, **more):
        return dict(name=name, kind=kind, disc=disc, dim=dim, coarse=coarse, refine=refine, **more)

    return [
        # a host Krylov loop on a small 2D problem: launches and copies are all it is
        case("cycle_2d_32", "cycle", "q1", 2, 2, 4, method=FLEXIBLE64),
        # the plain solver on a small plane problem, the reference's own method
        case("solve_2d_128_left", "solve", "q1", 2, 2, 6, method=LEFT, tol=1e-10),
        # the ordinary 3D diffusion solve, mixed precision: the benchmark's headline
        case("solve_3d_64_mixed", "solve", "q1", 3, 1, 6, method=MIXED),
        # the same equation as the reference solves it, on a mesh that is no power of two
        case("solve_3d_56_left", "solve", "q1", 3, 7, 3, method=LEFT),
        # block ILU smoothing (linear_smooth ilu)
        case("solve_3d_64_ilu", "solve", "q1", 3, 1, 6, method=MIXED, smoother="ilu"),
        # flow: stabilised Stokes with the Vanka smoother, plane and space
        case("stokes_2d_512_mixed", "solve", "stokes", 2, 2, 8, method=MIXED),
        case("stokes_3d_16_fp64", "solve", "stokes", 3, 2, 3, method=FLEXIBLE64),
        # quadratic elements, convection: long rows, many steps
        case("q2_3d_80_mixed", "solve", "q2", 3, 5, 4, method=MIXED),
        # the same with local refinement and hanging nodes
        case("q2_ball_40_fp64", "solve", "ball", 3, 5, 3, method=FLEXIBLE64),
        # a Newton step's assembly and residual, linear and quadratic elements
        case("newton_q1_3d_64", "newton", "q1", 3, 1, 6),
        case("newton_q2_3d_64", "newton", "q2", 3, 2, 5),
        # one step of a design loop: the largest mesh
        case("design_3d_96", "design", "q1", 3, 3, 5, method=MIXED),
    ]


def draw(rng):
    kind, disc = rng.choice([("cycle", "q1"), ("solve", "q1"), ("solve", "q1"), ("solve", "q1"),
                             ("solve", "stokes"), ("solve", "q2"), ("solve", "ball"),
                             ("newton", "q1"), ("newton", "q2"), ("design", "q1")])
    dim = 3 if disc == "ball" else rng.choice([2, 3, 3])
    smoother = "ilu" if (kind, disc) == ("solve", "q1") and rng.random() < 0.25 else ""
    # cells per dimension, smallest and largest
    lo, hi = {2: (16, 512), 3: (8, 64)}[dim]
    if disc in ("stokes", "q2") or smoother:
        lo, hi = {2: (16, 192), 3: (8, 16 if disc == "stokes" else 44)}[dim]
    if disc == "ball":
        lo, hi = 16, 40
    if (kind, disc, dim) == ("newton", "q2", 3):
        hi = 64
    n = lo * (hi / lo) ** rng.random()
    # a Stokes hierarchy ends above the one patch whose local system is singular
    coarsest = (2, 3, 5, 7) if disc == "stokes" else (1, 2, 3, 5, 7)
    sizes = [(c << r, c, r) for c in coarsest for r in range(2, 9) if lo <= c << r <= hi]
    near = sorted(sizes, key=lambda s: abs(s[0] / n - 1.0))[:4]
    _, coarse, refine = rng.choice(near)
    case = dict(kind=kind, disc=disc, dim=dim, coarse=coarse, refine=refine)
    if kind in ("cycle", "solve"):
        case["method"] = rng.choice([LEFT, FLEXIBLE64, MIXED] if kind == "solve" and disc == "q1"
                                    else [FLEXIBLE64, MIXED])
        case["mgtype"] = rng.choice("VVVWF" if disc == "q1" else "V")
    if smoother:
        case["smoother"] = smoother
    if kind == "newton":
        case["convection"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=2)
def _mesh(disc, dim, coarse, refine):
    """The levels of a mesh with coefficient 1: what does not depend on the seed."""
    if disc == "stokes":
        return structured_stokes(dim, coarse, refine)
    if disc == "q2":
        return structured_q2(dim, coarse, refine, eps=EPS, beta=BETA)
    if disc == "ball":
        return structured_q2_ball(coarse, refine, eps=EPS, beta=BETA)
    return structured_problem(dim, coarse, refine)


def _problem(case):
    return _mesh(case["disc"], case["dim"], case["coarse"], case["refine"])


def _kappa(case, seed):
    """Log-normal coefficient per finest element (Q2: per patch of cells, around EPS)."""
    q2 = case["disc"] == "q2"
    n = (case["coarse"] << case["refine"]) >> (1 if q2 else 0)
    z = np.random.default_rng([seed, 1]).normal(size=(n,) * case["dim"])
    return EPS * np.exp(0.25 * z) if q2 else np.exp(z)


def _vector(prob, seed, k):
    """Values in [-1, 1], 0 on the Dirichlet and hanging nodes."""
    fine = prob.finest
    v = np.random.default_rng([seed, k]).uniform(-1.0, 1.0, size=fine.ndof)
    v[fine.dirichlet] = 0.0
    for h in (fine.hn_edges, fine.hn_faces):
        if h is not None:
            v[h[:, 0]] = 0.0
    return v


def _rhs(case, prob, seed):
    if case["disc"] != "stokes":
        return _vector(prob, seed, 2)
    fine = prob.finest
    b = stokes_rhs(case["dim"], case["coarse"], case["refine"], seed).reshape(fine.n, fine.B)
    b[fine.dirichlet, 1:] = 0.0
    return b.ravel()


def _local_1d(h):
    """Mass and stiffness of a linear element of length h."""
    return (np.array([[2.0, 1.0], [1.0, 2.0]]) * (h / 6.0),
            np.array([[1.0, -1.0], [-1.0, 1.0]]) / h)


def _q1_local(dim, h):
    """Unit-coefficient stiffness of a cell of width h, nodes with x fastest."""
    m, s = _local_1d(h)
    out = 0.0
    for axis in range(dim):
        k = np.ones((1, 1))
        for d in range(dim):
            k = np.kron(k, s if d == axis else m)
        out = out + k
    return out


def _corners(dim):
    return [tuple(c) for c in np.ndindex(*(2,) * dim)]


def _q1_values(dim, kappa):
    """CSR values (columns ascending) of the Q1 matrix of per-cell kappa, the
    boundary rows and columns the identity's."""
    n = kappa.shape[0]
    local = _q1_local(dim, 1.0 / n)
    val = np.zeros((n + 1,) * dim + (3,) * dim)
    at = np.zeros((n + 1,) * dim + (3,) * dim, dtype=bool)
    for i, a in enumerate(_corners(dim)):
        rows = tuple(slice(x, x + n) for x in a)
        for j, b in enumerate(_corners(dim)):
            here = rows + tuple(y - x + 1 for x, y in zip(a, b))
            val[here] += local[i, j] * kappa
            at[here] = True
    inner = np.zeros((n + 1,) * dim, dtype=bool)
    inner[(slice(1, n),) * dim] = True
    padded = np.pad(inner, 1)
    for o in np.ndindex(*(3,) * dim):
        neighbour = padded[tuple(slice(k, k + n + 1) for k in o)]
        val[(Ellipsis,) + o] *= inner & neighbour
    val[(Ellipsis,) + (1,) * dim][~inner] = 1.0
    return val[at]


def _keys(case):
    """The solver keys (gb_params) the problems are solved with."""
    keys = dict(tol=case.get("tol", 1e-8), globaltol=1e-300, maxiter=200, gmressize=21, omega=0.8,
                mgtype=case.get("mgtype", "V"), smoother=case.get("smoother") or None)
    if case["disc"] == "stokes":
        keys.update(gmressize=31, omega=1.0)
    elif case["disc"] in ("q2", "ball"):
        keys.update(gmressize=31, omega=0.3, maxiter=600)
    elif case.get("smoother") == "ilu":
        keys.update(omega=1.0)
    return keys


def prepare(case, seed):
    prob = _problem(case)
    kind, q1 = case["kind"], case["disc"] == "q1"
    ctx = Context(0)
    state = dict(kind=kind, ctx=ctx, fine=prob.nlevels - 1, method=case.get("method"))
    if kind in ("solve", "cycle") and q1:  # assembled on the host, as a Gascoigne program has it
        pyramid = kappa_pyramid(prob.dim, _kappa(case, seed), prob.nlevels)
        prob = dataclasses.replace(prob, levels=[
            dataclasses.replace(lv, val=_q1_values(prob.dim, k))
            for lv, k in zip(prob.levels, pyramid)])
    ctx.load_problem(prob)
    ctx.set_params(**_keys(case))
    if kind == "solve":
        n = prob.finest.ndof
        state["b"] = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        state["x"] = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        state["b"][:] = _rhs(case, prob, seed)
    elif kind == "cycle":
        state.update(r=_vector(prob, seed, 2), x=ctx.vec(), y=ctx.vec())
    else:  # matrices assembled on the device from each new coefficient field
        if q1:
            for level, (cells, coords, parent) in enumerate(structured_meshes(prob)):
                ctx.set_mesh(level, prob.dim, cells, coords, parent)
        else:
            for level, (cells, parent) in enumerate(q2_meshes(prob)):
                ctx.set_mesh(level, prob.dim, cells, prob.levels[level].coord, parent, degree=2)
        state["kappa"] = torch.from_numpy(_kappa(case, seed).ravel()).cuda()
        state["beta"] = BETA[:prob.dim] if case.get("convection", not q1) else None
        state.update(u=ctx.vec(), b=ctx.vec(), y=ctx.vec(), w=ctx.vec())
        ctx.upload(state["fine"], state["b"], _vector(prob, seed, 2))
        ctx.upload(state["fine"], state["u"], _vector(prob, seed, 3))
    return state


# -------------------------------------------------------------------- call

def run(state):
    ctx, fine, kind = state["ctx"], state["fine"], state["kind"]
    if kind == "solve":
        x, _ = ctx.solve_host(state["b"], state["method"], out=state["x"], check=False)
        return x
    if kind == "cycle":
        ctx.upload(fine, state["y"], state["r"])
        ctx.zero(fine, state["x"])
        ctx.precondition(state["x"], state["y"],
                         GB_FP32 if state["method"] == MIXED else GB_FP64)
        return ctx.download(fine, state["x"])
    ctx.assemble_levels(state["kappa"], state["beta"])
    if kind == "newton":
        largest = ctx.newton_residual(state["y"], state["u"], state["b"])
        return {"residual": ctx.download(fine, state["y"]), "largest": largest}
    ctx.fgmres(state["u"], state["b"])
    value = ctx.functional(fine, state["u"], state["y"])
    ctx.adjoint_fgmres(state["w"], state["y"])
    return {"value": value, "gradient": ctx.coeff_gradient(fine, state["u"], state["w"])}


# -------------------------------------------------------------------- work

def _sizes(case):
    """(rows, matrix entries) per level, coarsest first."""
    out = []
    if case["disc"] == "ball":
        return [(lv.n, lv.nnzb) for lv in _problem(case).levels]
    for level in range(case["refine"]):
        n = (2 * case["coarse"]) << level
        per_axis = 4 * n + 1 if case["disc"] == "q2" else 3 * n + 1
        out.append(((n + 1) ** case["dim"], per_axis ** case["dim"]))
    return out


def work(case):
    """Each input read once and each result written once. A solve's matrix is
    counted once although every step reads it: the number of steps is not known
    beforehand."""
    sizes, dim = _sizes(case), case["dim"]
    block = dim + 1 if case["disc"] == "stokes" else 1
    rows, nnz = sizes[-1][0] * block, sum(s[1] for s in sizes) * block ** 2
    if case["kind"] in ("solve", "cycle"):
        return {"bytes": 8.0 * nnz + 16.0 * rows, "flops": 2.0 * nnz}
    q2 = case["disc"] == "q2"
    nloc, points = (3 ** dim, 3 ** dim) if q2 else (2 ** dim, 2 ** dim)
    cells = ((case["coarse"] << case["refine"]) >> q2) ** dim
    flops = 2.0 * cells * points * nloc ** 2 * (dim + 1)
    mesh = cells * (8.0 + 4.0 * nloc) + 8.0 * dim * rows
    moved = mesh + 8.0 * nnz + 24.0 * rows
    if case["kind"] == "design":  # two solves: the matrix once for each, and the gradient
        moved, flops = moved + 16.0 * nnz + 8.0 * cells, flops + 4.0 * nnz
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------- exact

class _Uniform:
    """-div(kappa grad) [+ beta . grad] on the uniform mesh of one level, by
    element products in 64 bits; zero boundary values."""

    def __init__(self, case, kappa, beta=None):
        self.dim, dev = case["dim"], "cuda" if torch.cuda.is_available() else "cpu"
        self.q2 = case["disc"] == "q2"
        n, step = kappa.shape[0], 2 if self.q2 else 1
        self.side = n * step + 1
        diffusion, convection = (_q2_local if self.q2 else _q1_both)(self.dim, 1.0 / n)
        self.kappa = torch.as_tensor(kappa, device=dev).reshape(-1, 1)
        self.local = torch.as_tensor(diffusion, device=dev)
        self.conv = None
        if beta is not None:
            self.conv = torch.as_tensor(sum(b * c for b, c in zip(beta, convection)), device=dev)
        grid = torch.arange(self.side ** self.dim, device=dev).reshape((self.side,) * self.dim)
        base = grid[tuple(slice(0, n * step, step) for _ in range(self.dim))].reshape(-1, 1)
        offs = grid[(slice(0, step + 1),) * self.dim].reshape(1, -1)
        self.nodes = base + offs
        inner = torch.zeros((self.side,) * self.dim, dtype=torch.float64, device=dev)
        inner[(slice(1, self.side - 1),) * self.dim] = 1.0
        self.inner = inner.reshape(-1)

    def _product(self, x):
        v = x[self.nodes]
        out = (v @ self.local.T) * self.kappa
        if self.conv is not None:
            out = out + v @ self.conv.T
        return torch.zeros_like(x).index_add_(0, self.nodes.reshape(-1), out.reshape(-1))

    def __call__(self, x):
        """A x, the boundary rows and columns the identity's."""
        return self._product(x * self.inner) * self.inner + x * (1.0 - self.inner)

    def form(self, x):
        """A x with the boundary columns kept, 0 on the boundary."""
        return self._product(x) * self.inner

    def diagonal(self):
        d = self.kappa * torch.diagonal(self.local)
        if self.conv is not None:
            d = d + torch.diagonal(self.conv)
        out = torch.zeros_like(self.inner).index_add_(0, self.nodes.reshape(-1), d.reshape(-1))
        return out * self.inner + (1.0 - self.inner)


def _q1_both(dim, h):
    return _q1_local(dim, h), []


def _q2_local(dim, h):
    """Unit-coefficient stiffness and the derivative matrices of a quadratic
    element of width h, nodes with x fastest, by the reference's three-point
    Gauss rule (its 12-digit weights)."""
    pts = np.array([0.11270166537925831148, 0.5, 0.88729833462074168852])
    wts = np.array([0.277777777778, 0.444444444444, 0.277777777778])
    f = np.stack([2 * (pts - 0.5) * (pts - 1), -4 * pts * (pts - 1), 2 * pts * (pts - 0.5)])
    g = np.stack([4 * pts - 3, -8 * pts + 4, 4 * pts - 1]) / h
    w = wts * h
    mass, stiff, slope = (f * w) @ f.T, (g * w) @ g.T, (f * w) @ g.T

    def tensor(axis, k):
        out = np.ones((1, 1))
        for d in reversed(range(dim)):
            out = np.kron(out, k if d == axis else mass)
        return out

    return (sum(tensor(a, stiff) for a in range(dim)), [tensor(a, slope) for a in range(dim)])


def _krylov(apply, diag, b, symmetric, steps=20000, tol=1e-13):
    """Conjugate gradients, or BiCGStab, with diagonal scaling; None if 20000
    steps do not reach the tolerance."""
    x, r = torch.zeros_like(b), b.clone()
    limit = tol * float(torch.linalg.norm(b))
    if symmetric:
        z = r / diag
        p, rz = z, torch.dot(r, z)
        for k in range(steps):
            q = apply(p)
            alpha = rz / torch.dot(p, q)
            x, r = x + alpha * p, r - alpha * q
            if k % 50 == 49 and float(torch.linalg.norm(r)) < limit:
                break
            z = r / diag
            old, rz = rz, torch.dot(r, z)
            p = z + (rz / old) * p
    else:
        shadow, rho, alpha, omega = r.clone(), 1.0, 1.0, 1.0
        p, v = torch.zeros_like(b), torch.zeros_like(b)
        for k in range(steps):
            old, rho = rho, torch.dot(shadow, r)
            p = r + (rho / old) * (alpha / omega) * (p - omega * v)
            ph = p / diag
            v = apply(ph)
            alpha = rho / torch.dot(shadow, v)
            s = r - alpha * v
            sh = s / diag
            t = apply(sh)
            omega = torch.dot(t, s) / torch.dot(t, t)
            x, r = x + alpha * ph + omega * sh, s - omega * t
            if k % 20 == 19 and not float(torch.linalg.norm(r)) > limit:
                break
    good = float(torch.linalg.norm(b - apply(x))) < 20 * limit
    return x if good else None


def _stokes_exact(prob, b):
    """Dense solve of a small Stokes system; the pressure's mean taken out."""
    fine = prob.finest
    if fine.ndof > 20000:
        return None
    block = fine.B
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rows = torch.as_tensor(np.repeat(np.arange(fine.n), np.diff(fine.rowptr)), device=dev)
    cols = torch.as_tensor(fine.col, device=dev)
    a = torch.zeros(fine.ndof, fine.ndof, dtype=torch.float64, device=dev)
    val = torch.as_tensor(fine.val, device=dev).reshape(-1, block, block)
    for i in range(block):
        for j in range(block):
            a[rows * block + i, cols * block + j] = val[:, i, j]
    p = torch.zeros(fine.ndof, dtype=torch.float64, device=dev)
    p[::block] = 1.0 / fine.n
    a.addr_(p, p, alpha=float(fine.n))  # the constant pressure is the matrix's kernel
    x = torch.linalg.solve(a, torch.as_tensor(b, device=dev)).cpu().numpy()
    x[::block] -= np.dot(fine.pf_weights, x[::block]) / fine.pf_domain
    return x


def _smooth(op, diag, x, b, sweeps, omega):
    for _ in range(sweeps):
        x = x + omega * (b - op(x)) / diag
    return x


def _cycle(ops, level, b, omega, kind, first):
    """One V, W or F cycle of Jacobi smoothing from zero (or `first`)."""
    op, x = ops[level], torch.zeros_like(b) if first is None else first
    diag = op.diagonal()
    if level == 0:
        return _smooth(op, diag, x, b, 10, omega)
    x = _smooth(op, diag, x, b, 2, omega)
    coarse = ops[level - 1]
    between = torch.zeros(op.side, coarse.side, dtype=torch.float64, device=b.device)
    i = torch.arange(coarse.side, device=b.device)
    between[2 * i, i] = 1.0
    between[2 * i[:-1] + 1, i[:-1]] = 0.5
    between[2 * i[:-1] + 1, i[1:]] = 0.5

    def axes(v, side, m):
        v = v.reshape((side,) * op.dim)
        for d in range(op.dim):
            v = torch.movedim(torch.tensordot(m, v, dims=([1], [d])), 0, d)
        return v.reshape(-1)

    r = axes(b - op(x), op.side, between.T.contiguous()) * coarse.inner
    e = _cycle(ops, level - 1, r, omega, kind, None)
    if kind == "W":
        e = _cycle(ops, level - 1, r, omega, kind, e)
    x = x + axes(e, coarse.side, between) * op.inner
    return _smooth(op, diag, x, b, 2, omega)


def exact(case, seed):
    prob, kind, q1 = _problem(case), case["kind"], case["disc"] == "q1"
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["disc"] == "stokes":
        return _stokes_exact(prob, _rhs(case, prob, seed))
    if case["disc"] == "ball":
        fine = prob.finest
        a = torch.sparse_csr_tensor(torch.as_tensor(fine.rowptr), torch.as_tensor(fine.col),
                                    torch.as_tensor(fine.val), size=(fine.n, fine.n)).to(dev)
        diag = torch.as_tensor(fine.val[fine.diag], device=dev)
        b = torch.as_tensor(_rhs(case, prob, seed), device=dev)
        x = _krylov(lambda v: torch.mv(a, v), diag, b, False)
        return None if x is None else x.cpu().numpy()
    kappa = _kappa(case, seed)
    if kind == "cycle":
        if case.get("mgtype", "V") == "F":
            return None  # its visiting order is a convention of its own
        ops = [_Uniform(case, k) for k in kappa_pyramid(prob.dim, kappa, prob.nlevels)]
        r = torch.as_tensor(_vector(prob, seed, 2), device=dev)
        return _cycle(ops, prob.nlevels - 1, r, 0.8, case.get("mgtype", "V"), None).cpu().numpy()
    if kind == "solve":
        op = _Uniform(case, kappa) if q1 else _Uniform(case, np.full_like(kappa, EPS), BETA)
        x = _krylov(op, op.diagonal(), torch.as_tensor(_rhs(case, prob, seed), device=dev), q1)
        return None if x is None else x.cpu().numpy()
    op = _Uniform(case, kappa)
    b = torch.as_tensor(_vector(prob, seed, 2), device=dev)
    if kind == "newton":
        if case.get("convection", not q1):
            if q1:
                return None
            op = _Uniform(case, kappa, BETA)
        y = (b - op.form(torch.as_tensor(_vector(prob, seed, 3), device=dev))) * op.inner
        return {"residual": y.cpu().numpy(), "largest": float(y.abs().max())}
    u = _krylov(op, op.diagonal(), b, True)
    if u is None:
        return None
    h = 1.0 / kappa.shape[0]
    mass = np.ones((1, 1))
    for _ in range(prob.dim):
        mass = np.kron(mass, _local_1d(h)[0])
    cell = u[op.nodes]
    mu = cell @ torch.as_tensor(mass, device=dev).T
    value = float((cell * mu).sum())
    slope = 2.0 * torch.zeros_like(u).index_add_(0, op.nodes.reshape(-1), mu.reshape(-1)) * op.inner
    w = _krylov(op, op.diagonal(), slope, True)
    if w is None:
        return None
    gradient = -((w[op.nodes] @ op.local) * cell).sum(1)
    return {"value": value, "gradient": gradient.cpu().numpy()}
