"""The work a user of this package has it do, as cases that can be timed one by one.

Five kinds, each through the public classes of :mod:`parmoon_cmg_b200.system`:

``solve``     a stationary problem as the reference's CD2D / CD3D mains run it: assemble every
              multigrid level, copy the right-hand side to the host, solve from a host start
              vector, solution back on the host;
``product``   one FP64 product y = A x on device vectors, from the CSR entries or matrix-free;
``assemble``  assembly with coefficients tabulated at the quadrature points (every example whose
              BilinearCoeffs vary in space), then one product with the new matrix;
``tcd``       one theta-scheme step of a time-dependent problem: stiffness matrix and right-hand
              side at the new time, system matrix, solve from the previous solution;
``batch``     many independent problems submitted, advanced together, fetched and released,
              stationary (``steps`` 0) or a few time steps each.

Meshes are uniform refinements of the unit square or cube (``n0`` cells per side on the
coarsest of ``levels`` levels), optionally deformed (``warp``) so that cells are not affine.
Everything else -- convection direction, diffusion, tables, vectors, initial values -- comes
from the seed.
"""
import functools
import math

import numpy as np
import torch

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.serving import default_params
from parmoon_cmg_b200.system import (GALERKIN, SUPG, Batch, Context, TSystemCD2D, TSystemCD3D, TSystemTCD2D,
                                     TSystemTCD3D, coeffs, solver_params)
from parmoon_cmg_b200.workloads import StructureCache, dofs, hierarchy_shape

TAU, THETA = 1e-3, (0.5, 0.5, 0.5, 0.5)  # Crank-Nicolson, the time step of the TCD2D workload


def listed():
    return [
        # the smallest stationary problem in use (4,225 unknowns): launches and latency count
        dict(name="cd2d_q1_64_f64", kind="solve", dim=2, order=1, n0=4, levels=5, supg=True, precision=0),
        # an ordinary 2D problem in the mixed form, a mesh that is not a power of two
        dict(name="cd2d_q2_192_mixed", kind="solve", dim=2, order=2, n0=3, levels=7, supg=True, precision=1),
        # an ordinary 3D problem with trilinear elements
        dict(name="cd3d_q1_48_mixed", kind="solve", dim=3, order=1, n0=3, levels=5, supg=True, precision=1),
        # the benchmark problem in its two forms
        dict(name="cd3d_q2_32_mixed", kind="solve", dim=3, order=2, n0=2, levels=5, supg=False, precision=1),
        dict(name="cd3d_q2_32_f64", kind="solve", dim=3, order=2, n0=2, levels=5, supg=False, precision=0),
        # one matrix-vector product, matrix larger than L2; and without the matrix
        dict(name="product_csr_q2_32", kind="product", dim=3, order=2, n0=32, levels=1, form=0),
        dict(name="product_mf_q2_32", kind="product", dim=3, order=2, n0=32, levels=1, form=1),
        # variable coefficients on deformed hexahedra, and 2D SUPG with variable coefficients
        dict(name="assemble_3d_q2_24_table", kind="assemble", dim=3, order=2, n0=24, levels=1, supg=False, warp=True),
        dict(name="assemble_2d_q2_160_table", kind="assemble", dim=2, order=2, n0=160, levels=1, supg=True, warp=False),
        # a time step of the rotating-convection workload, one system
        dict(name="tcd2d_q2_128_f64", kind="tcd", dim=2, order=2, n0=2, levels=7, precision=0),
        # a request queue's worth of independent solves of mixed sizes, multicolour SSOR
        dict(name="batch_cd2d_40", kind="batch", count=40, n_min=16, n_max=128, mix=1, steps=0),
        # independent time-dependent problems advanced together, damped Jacobi
        dict(name="batch_tcd2d_16", kind="batch", count=16, n_min=128, n_max=128, mix=2, steps=6),
    ]


def draw(rng):
    def log_between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def shape(n):
        # n cells per side as n0 * 2^(levels - 1) with 2 <= n0 <= 5
        levels = max(2, int(math.floor(math.log2(n / 2.0))) + 1)
        n0 = max(2, min(5, int(round(n / 2 ** (levels - 1)))))
        return dict(n0=n0, levels=levels)

    kind = rng.choice(["solve", "solve", "solve", "product", "assemble", "assemble", "tcd", "batch"])
    dim, order = rng.choice([2, 3]), rng.choice([1, 2])
    if kind == "tcd" and dim == 3:
        order = 1  # damped Jacobi does not smooth the mass matrix of triquadratic elements
    if kind in ("solve", "tcd"):
        n = log_between(16, 192 // order) if dim == 2 else log_between(8, 48 if order == 1 else 24)
        case = dict(kind=kind, dim=dim, order=order, precision=rng.choice([0, 1]), **shape(n))
        if kind == "solve":
            case["supg"] = order == 1 or dim == 2 or rng.random() < 0.5
        return case
    if kind == "product":
        n = log_between(256 // order, 400 // order) if dim == 2 else log_between(36 // order, 64 // order)
        form = rng.choice([0, 1]) if (dim, order) == (3, 2) else 0
        return dict(kind=kind, dim=dim, order=order, n0=n, levels=1, form=form)
    if kind == "assemble":
        n = log_between(16, 240 // order) if dim == 2 else log_between(5, 48 // order)
        return dict(kind=kind, dim=dim, order=order, n0=n, levels=1, supg=rng.random() < 0.5, warp=rng.random() < 0.5)
    if rng.random() < 0.5:
        return dict(kind="batch", count=log_between(4, 40), n_min=16, n_max=rng.choice([48, 64, 96, 128]),
                    mix=rng.randrange(1000), steps=0)
    n = rng.choice([32, 48, 64, 96])
    return dict(kind="batch", count=log_between(2, 16), n_min=n, n_max=n, mix=2, steps=rng.randint(2, 6))


# ---------------------------------------------------------------------------
# problems
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _hierarchy(dim, order, n0, levels):
    return mesh.structured_hierarchy(dim, order, n0, levels)


def _cells(case):
    return case["n0"] * 2 ** (case["levels"] - 1)


def _warp(xyz):
    """A smooth deformation of the unit square or cube that keeps its boundary in place."""
    s = np.prod(np.sin(np.pi * xyz), axis=-1, keepdims=True)
    return xyz + s * np.array([0.06, -0.05, 0.04])[:xyz.shape[-1]]


def _spaces(case):
    spaces, parents = _hierarchy(case["dim"], case["order"], case["n0"], case["levels"])
    if case.get("warp"):
        d = case["dim"]
        spaces = [dict(s, coords=np.ascontiguousarray(_warp(s["coords"].reshape(-1, d)).reshape(-1))) for s in spaces]
    return spaces, parents


def _problem(case, seed):
    """Constant coefficients of a stationary problem: a direction near the diagonal of the
    domain, diffusion in the range damped Jacobi smooths on the case's meshes."""
    rng = np.random.default_rng(seed)
    dim = case["dim"]
    b = 1.0 + rng.uniform(-0.4, 0.4, dim)
    b /= np.linalg.norm(b)
    small = (dim, case["order"]) == (2, 1) and _cells(case) <= 64
    eps = (1e-3 if small else 1e-2) * math.exp(rng.uniform(0.0, 0.5))
    return dict(eps=eps, b=tuple(float(v) for v in b), f=float(rng.uniform(0.5, 1.5)), c=0.0,
                delta0=1.0 if case.get("supg") else 1.0 / 3.0)


def _table(xyz, seed):
    """(eps, b1, b2, b3, c, f) at points: smooth fields of the seed."""
    rng = np.random.default_rng(seed)
    p, q = rng.uniform(0.0, 2.0 * np.pi, 8), rng.uniform(0.5, 1.5, 8)
    x, y = xyz[..., 0], xyz[..., 1]
    z = xyz[..., 2] if xyz.shape[-1] == 3 else np.zeros_like(x)
    out = np.zeros(xyz.shape[:-1] + (6,))
    out[..., 0] = 1e-2 * (1.0 + 0.5 * np.sin(q[0] * x + 2.0 * y + z + p[0]))
    out[..., 1] = q[1] * (0.5 - y) + 0.2 * np.cos(3.0 * z + p[1])
    out[..., 2] = q[2] * (x - 0.5) + 0.2 * np.sin(2.0 * z + p[2])
    out[..., 3] = 0.25 * np.cos(q[3] * x + y + p[3]) if xyz.shape[-1] == 3 else 0.0
    out[..., 4] = 0.1 * (1.0 + np.sin(q[4] * x * y + p[4]))
    out[..., 5] = 1.0 + 0.5 * np.sin(q[5] * x + 3.0 * y - z + p[5])
    return out


def _bump(xy, rng):
    c = rng.uniform(0.25, 0.45, xy.shape[1])
    return np.exp(-((xy - c) ** 2).sum(1) / (2 * 0.08 ** 2))


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _instances(case, seed):
    """The instances of a batch: meshes fixed by the case, coefficients from the seed."""
    sizes, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        order = 2 if case["steps"] else (1 if sizes.random() < 0.5 else 2)
        ang = rng.uniform(0, 2 * math.pi)
        eps = 10.0 ** (rng.uniform(-5, -2) if case["steps"] else rng.uniform(-6, -1))
        out.append(dict(n=hierarchy_shape(n)[2], order=order, eps=eps, b=(math.cos(ang), math.sin(ang))))
    return out


# ---------------------------------------------------------------------------
# what a program has in hand before the call, and the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "solve":
        spaces, parents = _spaces(case)
        cls = TSystemCD2D if case["dim"] == 2 else TSystemCD3D
        # a Galerkin fine level keeps SUPG coarse-grid operators, as in the benchmark problem
        S = cls(spaces, parents, disctype=SUPG if case["supg"] else GALERKIN, coarse_disctype=SUPG)
        S.Init(coeffs(**_problem(case, seed)))
        state.update(S=S, sol=_pinned(S.N_DOF), rhs=_pinned(S.N_DOF),
                     prm=solver_params(precision=case["precision"], stop_rule=1, red_factor=1e-10, maxit=300))
    elif kind in ("product", "assemble"):
        spaces, parents = _spaces(case)
        cls = TSystemCD2D if case["dim"] == 2 else TSystemCD3D
        S = cls(spaces, parents, disctype=SUPG if case.get("supg") else GALERKIN)
        if kind == "product":
            S.Init(coeffs(**_problem(case, seed)))
            S.Assemble()
        else:
            xq = S.ctx.quadrature_points(S.sids[0], spaces[0]["n_cells"], case["dim"])
            S.Init(coeffs(_lib.COEFF_TABLE, poly_degree=case["order"]), table=[_table(xq, seed)])
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        x = torch.rand(S.N_DOF, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        x[S.N_Active:] = 0.0  # boundary rows are identity rows: the product is of the inner unknowns
        state.update(S=S, x=x, y=torch.zeros_like(x), sol=_pinned(S.N_DOF), rhs=_pinned(S.N_DOF))
    elif kind == "tcd":
        spaces, parents = _spaces(case)
        cls = TSystemTCD2D if case["dim"] == 2 else TSystemTCD3D
        S = cls(spaces, parents)
        rng = np.random.default_rng(seed)
        S.Init(_tcd_coeffs(case["dim"], 10.0 ** rng.uniform(-4, -2), rng.uniform(0.0, 0.5)))
        u0 = _bump(mesh.dof_coords(spaces[-1]), rng)
        S.AssembleMRhs(u0)
        state.update(S=S, u0=u0, sol=_pinned(S.N_DOF),
                     prm=solver_params(precision=case["precision"], stop_rule=1, red_factor=1e-10, maxit=300))
    else:
        steps = case["steps"]
        prm = default_params()
        if steps:
            prm = solver_params(smoother=1, omega=0.8, stop_rule=1, red_factor=1e-10, maxit=500)
        B = Batch(prm, Context())
        cache, work = StructureCache(B), _instances(case, seed)
        for w in work:
            w["structure"], w["n_dof"] = cache.get(2, w["order"], w["n"])
        if steps:
            rng = np.random.default_rng(seed + 1)
            for w in work:
                sp = _hierarchy(2, w["order"], hierarchy_shape(w["n"])[1], hierarchy_shape(w["n"])[0])[0][-1]
                w["u0"] = _bump(mesh.dof_coords(sp), rng)
                w["u0"][sp["n_active"]:] = 0.0
        state.update(B=B, work=work)
    return state


def _tcd_coeffs(dim, eps, f):
    if dim == 2:
        return coeffs(_lib.COEFF_ROTATING, eps=eps, f=f)
    return coeffs(_lib.COEFF_CONSTANT, eps=eps, b=(0.5, 0.3, -0.4), f=f)


def run(state):
    kind = state["case"]["kind"]
    if kind == "batch":
        return _run_batch(state)
    S = state["S"]
    if kind == "solve":
        state["sol"][:] = 0.0
        S.Assemble(state["sol"], state["rhs"])
        S.Solve(state["sol"], state["rhs"], state["prm"])
        return {"rhs": state["rhs"], "sol": state["sol"]}
    if kind == "tcd":
        state["sol"][:] = state["u0"]
        S.AssembleARhs()
        S.Step(state["sol"], TAU, *THETA, params=state["prm"])
        return state["sol"]
    out = {"y": state["y"]}
    form = state["case"].get("form", 0)
    if kind == "assemble":
        S.Assemble(state["sol"], state["rhs"])
        out["rhs"] = state["rhs"]
    S.ctx.check(S.ctx.lib.cdgpu_apply_fp64_device(S.ctx.h, S.sids[-1], form, state["x"].data_ptr(),
                                                  state["y"].data_ptr()))
    return out


def _run_batch(state):
    B, steps = state["B"], state["case"]["steps"]
    slots = []
    for w in state["work"]:
        if steps:
            co = coeffs(_lib.COEFF_ROTATING, eps=w["eps"], f=0.0)
            slots.append(B.submit_tcd(w["structure"], co, TAU, *THETA, w["u0"]))
        else:
            co = coeffs(eps=w["eps"], b=w["b"], f=1.0, poly_degree=w["order"])
            slots.append(B.submit(w["structure"], co, SUPG))
    if steps:
        for _ in range(steps):
            B.tcd_step(8)
    else:
        B.run(8)
    out = [B.fetch(s, w["n_dof"])[0] for s, w in zip(slots, state["work"])]
    for s in slots:
        B.release(s)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(dim, order, n):
    """(cells, unknowns, nonzeros, local unknowns) of a uniform mesh."""
    per_dim = 3 * n + 1 if order == 1 else 8 * n + 1  # couplings of a one-dimensional mesh
    return n ** dim, (order * n + 1) ** dim, per_dim ** dim, (order + 1) ** dim


def work(case):
    """Bytes: the mesh, coefficient tables and vectors that come in, the matrix where one is
    assembled, the vectors that go out, each once.  Flops: the local forms (20 per cell, Gauss
    point and local entry on general cells, 2 per local entry and tensor on affine ones), two
    per nonzero and product; a solve counts ten preconditioned iterations of six products each
    on the finest level and a hierarchy that adds a geometric series, a time step five."""
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for w in _instances(case, 0):
            sub = dict(dim=2, order=w["order"], n0=w["n"], levels=1)
            one = work(dict(sub, kind="tcd" if case["steps"] else "solve"))
            b += one["bytes"] * max(1, case["steps"])
            f += one["flops"] * max(1, case["steps"])
        return dict(bytes=b, flops=f)
    dim, order = case["dim"], case["order"]
    cells, n, nnz, nbf = _sizes(dim, order, _cells(case))
    if kind == "product":
        if case["form"] == 1:
            return dict(bytes=cells * (4.0 * nbf + 8 * 10) + 16.0 * n, flops=cells * 2.0 * 1296)
        return dict(bytes=12.0 * nnz + 20.0 * n, flops=2.0 * nnz)
    nq = ((order + 2) if order == 2 else 3) ** dim
    geometry = cells * (8.0 * 2 ** dim * dim + 4.0 * nbf)
    if kind == "assemble":
        return dict(bytes=geometry + cells * nq * 48.0 + 20.0 * nnz + 24.0 * n,
                    flops=cells * nq * nbf * nbf * 20.0 + 2.0 * nnz)
    series = 1.0 / (1.0 - 0.5 ** dim)
    iterations = 10 if kind == "solve" else 5
    local = cells * nbf * nbf * 2.0 * 10
    return dict(bytes=geometry * series + 8.0 * nnz * series + 24.0 * n,
                flops=series * (local + iterations * 6 * 2.0 * nnz))


# ---------------------------------------------------------------------------
# the same outputs in 64 bits by dense and sparse-free means: local forms by Gauss quadrature,
# block elimination over the layers of cells
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return x, w


def _element(dim, order):
    """Gauss points, weights, basis values, gradients, second derivatives (x fastest)."""
    x, w = _gauss(3 if order == 1 else 4)
    if order == 1:
        v = np.stack([0.5 * (1 - x), 0.5 * (1 + x)], 1)
        d, h = np.stack([0 * x - 0.5, 0 * x + 0.5], 1), np.zeros((len(x), 2))
    else:
        v = np.stack([0.5 * x * (x - 1), 1 - x * x, 0.5 * x * (x + 1)], 1)
        d, h = np.stack([x - 0.5, -2 * x, x + 0.5], 1), np.tile([1.0, -2.0, 1.0], (len(x), 1))
    der = [v, d, h]

    def product(kinds):  # kinds[a]: derivative order in direction a
        t = der[kinds[0]]
        for k in kinds[1:]:
            t = np.einsum("pi,qj->pqij", der[k], t).reshape(len(der[k]) * t.shape[0], -1)
        return t

    unit = np.eye(dim, dtype=int)
    pts = np.stack(np.meshgrid(*[x] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
    wts = np.prod(np.stack(np.meshgrid(*[w] * dim, indexing="ij"), -1).reshape(-1, dim), 1)
    phi = product([0] * dim)
    dphi = np.stack([product(unit[a]) for a in range(dim)], -1)
    hphi = np.stack([np.stack([product(unit[a] + unit[e]) for e in range(dim)], -1) for a in range(dim)], -2)
    return pts, wts, phi, dphi, hphi


class _Forms:
    """Local forms of cells with vertices V (cells x vertices x dim, the order of the mesh
    module): physical gradients, weights and, in 2D, Laplacians at the Gauss points."""

    def __init__(self, dim, order, V):
        pts, wts, phi, dphi, hphi = _element(dim, order)
        t = functools.partial(torch.tensor, dtype=torch.float64, device=_device())
        corner = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                           [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])[:2 ** dim, :dim]
        one = 1 + corner[None] * pts[:, None, :]  # points x vertices x dim
        N = np.prod(one, -1) / 2 ** dim
        dN = np.stack([corner[None, :, a] * np.prod(np.delete(one, a, -1), -1) for a in range(dim)], -1) / 2 ** dim
        V = t(V)
        J = torch.einsum("qva,cvr->cqra", t(dN), V)  # dx_r / dxi_a
        Ji = torch.linalg.inv(J)
        self.x = torch.einsum("qv,cvr->cqr", t(N), V)
        self.w = t(wts) * torch.linalg.det(J).abs()
        self.phi = t(phi)
        self.g = torch.einsum("qia,cqar->cqir", t(dphi), Ji)
        pairs = [(0, 2), (1, 3)] if dim == 2 else [(0, 6), (1, 7), (2, 4), (3, 5)]
        self.h = torch.stack([(V[:, q] - V[:, p]).norm(dim=1) for p, q in pairs]).amax(0)  # longest diagonal
        self.lap = None
        if dim == 2:
            mixed = 0.25 * (V[:, 0] - V[:, 1] + V[:, 2] - V[:, 3])  # d2x / dxi deta
            H = t(hphi)[None] - torch.einsum("cqir,cr,ae->cqiae", self.g, mixed, t([[0.0, 1.0], [1.0, 0.0]]))
            self.lap = torch.einsum("cqar,cqiae,cqer->cqi", Ji, H, Ji)

    def streamline(self, k, degree, delta0):
        """The SUPG parameter at the Gauss points, nu h (coth a - 1 / a) / (2 |b|)."""
        nb = k[..., 1:4].norm(dim=-1).clamp_min(1e-300)
        nu, h = 1.0 / degree, self.h[:, None]
        a = nu * nb * h / (2 * k[..., 0])
        d = nu * h * (1 / torch.tanh(a) - 1 / a) / (2 * nb)
        return torch.where(k[..., 1:4].norm(dim=-1) > 0, d * delta0, torch.zeros_like(d))

    def test_and_trial(self, k, supg, degree, delta0):
        """Per point: test function of the residual terms, and the residual's trial part."""
        b = k[..., 1:1 + self.g.shape[-1]]
        bg = torch.einsum("cqir,cqr->cqi", self.g, b)
        trial = bg + k[..., 4:5] * self.phi
        test, extra = self.phi.expand_as(bg), None
        if supg:
            extra = self.streamline(k, degree, delta0)[..., None] * bg
            res = trial - (k[..., 0:1] * self.lap if self.lap is not None else 0.0)
        else:
            res = trial
        return test, trial, extra, res

    def matrices(self, k, supg, degree, delta0):
        """Local matrices and right-hand sides."""
        test, trial, extra, res = self.test_and_trial(k, supg, degree, delta0)
        A = torch.einsum("cq,cqir,cqjr->cij", self.w * k[..., 0], self.g, self.g)
        A += torch.einsum("cq,cqi,cqj->cij", self.w, test, trial)
        F = torch.einsum("cq,cqi->ci", self.w * k[..., 5], test)
        if extra is not None:
            A += torch.einsum("cq,cqi,cqj->cij", self.w, extra, res)
            F = F + torch.einsum("cq,cqi->ci", self.w * k[..., 5], extra)
        return A, F

    def products(self, k, supg, degree, delta0, xc):
        """Local products A_c x_c and right-hand sides, without the local matrices."""
        test, trial, extra, res = self.test_and_trial(k, supg, degree, delta0)
        y = torch.einsum("cqir,cqr->ci", self.g,
                         (self.w * k[..., 0])[..., None] * torch.einsum("cqjr,cj->cqr", self.g, xc))
        y += torch.einsum("cq,cqi->ci", self.w * torch.einsum("cqj,cj->cq", trial, xc), test)
        F = torch.einsum("cq,cqi->ci", self.w * k[..., 5], test)
        if extra is not None:
            y += torch.einsum("cq,cqi->ci", self.w * torch.einsum("cqj,cj->cq", res, xc), extra)
            F = F + torch.einsum("cq,cqi->ci", self.w * k[..., 5], extra)
        return y, F

    def mass(self):
        return torch.einsum("cq,qi,qj->cij", self.w, self.phi, self.phi)


class _Grid:
    """Lattice of a uniform mesh: nodes of every cell, and the numbering of the outputs (inner
    nodes, then boundary nodes, lexicographic in each class)."""

    def __init__(self, dim, order, n):
        self.dim, self.order, self.n = dim, order, n
        m = self.m = order * n + 1
        cell = np.stack(np.meshgrid(*[np.arange(n)] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
        loc = np.stack(np.meshgrid(*[np.arange(order + 1)] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
        stride = m ** np.arange(dim)
        self.nodes = ((order * cell[:, None] + loc[None]) * stride).sum(-1)
        idx = np.stack(np.meshgrid(*[np.arange(m)] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
        edge = ((idx == 0) | (idx == m - 1)).any(1)
        self.output_order = np.concatenate([np.flatnonzero(~edge), np.flatnonzero(edge)])
        self.n_active = int((~edge).sum())
        corner = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0],
                           [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])[:2 ** dim, :dim]
        self.cell, self.corner = cell, corner

    def vertices(self, cells=None):
        c = self.cell if cells is None else self.cell[cells]
        return (c[:, None] + self.corner[None]) / self.n

    def scatter(self, local):
        """Sum of local vectors (cells x local unknowns) over the lattice."""
        out = torch.zeros(self.m ** self.dim, dtype=torch.float64, device=local.device)
        nodes = torch.as_tensor(self.nodes.reshape(-1), device=local.device)
        return out.index_add_(0, nodes, local.reshape(-1))

    def give(self, lattice):
        return lattice.cpu().numpy()[self.output_order]

    def take(self, x):
        out = np.empty(len(x))
        out[self.output_order] = x
        return torch.tensor(out, device=_device())


class _Layers:
    """LU of the matrix of a uniform mesh on its inner nodes, by blocks: block k holds the node
    layers order*k + 1 .. order*(k + 1) of the last direction.  local(k): local matrices of the
    cells of layer k (cells or 1 x nbf x nbf)."""

    def __init__(self, grid, local, uniform):
        g, p, n, m = grid, grid.order, grid.n, grid.m
        self.g = g
        plane = m ** (g.dim - 1)
        idx = np.arange(plane)
        inner = np.ones(plane, bool)
        for a in range(g.dim - 1):
            q = idx // m ** a % m
            inner &= (q > 0) & (q < m - 1)
        self.inner = np.flatnonzero(inner)
        ni = self.ni = len(self.inner)
        per = n ** (g.dim - 1)
        # rows of layer-k cells in (face below, block k): position in (p + 1) * ni, -1 outside
        pos = -np.ones(plane, np.int64)
        pos[self.inner] = np.arange(ni)
        first = g.nodes[:per]
        where = torch.tensor(np.where(pos[first % plane] < 0, -1, first // plane * ni + pos[first % plane]),
                             device=_device())
        size = (p + 1) * ni
        pair = where[:, :, None] * size + where[:, None, :]
        keep = (where[:, :, None] >= 0) & (where[:, None, :] >= 0)

        def block(k):
            A = torch.zeros(size * size, dtype=torch.float64, device=_device())
            loc = local(k).expand(per, -1, -1)
            return A.index_add_(0, pair[keep], loc[keep]).view(size, size)

        self.S, self.L, self.W = [], [], []
        E = block(0)
        face = slice((p - 1) * ni, p * ni)
        rows_of = [p * ni] * (n - 1) + [(p - 1) * ni]  # the last node layer is the boundary
        self.blocks = n if p > 1 else n - 1
        for k in range(self.blocks):
            rows = rows_of[k]
            D = E[ni:ni + rows, ni:ni + rows].clone()
            if k + 1 < n:
                N = E if uniform else block(k + 1)
                D[face, face] += N[:ni, :ni]
            if k > 0:
                Lk = E[ni:ni + rows, :ni].clone()  # coupling to the last layer of block k - 1
                D -= Lk @ self.W[-1][face, :rows]
                self.L.append(Lk)
            lu = torch.linalg.lu_factor(D)
            self.S.append(lu)
            if k + 1 < self.blocks:
                U = torch.zeros(rows, rows_of[k + 1], dtype=torch.float64, device=_device())
                U[face] = N[:ni, ni:ni + rows_of[k + 1]]
                self.W.append(torch.linalg.lu_solve(*lu, U))
                E = N
        self.face = face

    def solve(self, lattice):
        """Solution on the lattice (zero on the boundary) of a right-hand side on the lattice."""
        p, plane = self.g.order, self.g.m ** (self.g.dim - 1)
        f = lattice.view(-1, plane)[1:-1][:, torch.as_tensor(self.inner, device=lattice.device)].reshape(-1)
        size, y = p * self.ni, []
        for k in range(self.blocks):
            r = f[k * size:(k + 1) * size].clone()
            if k > 0:
                r -= self.L[k - 1] @ y[-1][self.face]
            y.append(torch.linalg.lu_solve(*self.S[k], r[:, None])[:, 0])
        for k in range(self.blocks - 2, -1, -1):
            y[k] = y[k] - self.W[k] @ y[k + 1]
        out = torch.zeros_like(lattice).view(-1, plane)
        sub = torch.cat(y).view(-1, self.ni)
        out[1:-1, torch.as_tensor(self.inner, device=lattice.device)] = sub
        return out.view(-1)


def _constant(p, forms):
    k = [p["eps"], *p["b"], *([0.0] * (3 - len(p["b"]))), p["c"], p["f"]]
    return torch.tensor(k, dtype=torch.float64, device=_device()).expand(*forms.w.shape, 6)


def _zero_boundary(grid, lattice):
    out = lattice.clone()
    out[torch.as_tensor(grid.output_order[grid.n_active:], device=lattice.device)] = 0.0
    return out


def _exact_stationary(dim, order, n, p, supg, degree):
    grid = _Grid(dim, order, n)
    forms = _Forms(dim, order, grid.vertices([0]))  # every cell is the same
    A, F = forms.matrices(_constant(p, forms), supg, degree, p["delta0"])
    rhs = _zero_boundary(grid, grid.scatter(F.expand(n ** dim, -1).contiguous()))
    sol = _Layers(grid, lambda k: A, True).solve(rhs)
    return grid.give(rhs), grid.give(sol)


def _exact_steps(dim, order, n, eps, f, u0, steps):
    """Crank-Nicolson steps of the time-dependent problem from the nodal values u0."""
    grid = _Grid(dim, order, n)
    per = n ** (dim - 1)
    if dim == 2:
        forms = _Forms(dim, order, grid.vertices())
        k = torch.zeros(*forms.w.shape, 6, dtype=torch.float64, device=_device())
        k[..., 0], k[..., 5] = eps, f
        k[..., 1], k[..., 2] = 0.5 - forms.x[..., 1], forms.x[..., 0] - 0.5
    else:
        forms = _Forms(dim, order, grid.vertices([0]))
        k = _constant(dict(eps=eps, b=(0.5, 0.3, -0.4), c=0.0, f=f), forms)
    A, F = forms.matrices(k, False, 1, 1.0)
    M = forms.mass()
    t1, t2, t3, t4 = (TAU * t for t in THETA)
    S, K = M + t1 * A, M - t2 * A
    uniform = S.shape[0] == 1
    lay = _Layers(grid, lambda j: S if uniform else S[j * per:(j + 1) * per], uniform)
    rhs_f = grid.scatter(((t3 + t4) * F).expand(n ** dim, -1).contiguous())
    nodes = torch.as_tensor(grid.nodes, device=_device())
    u = _zero_boundary(grid, grid.take(u0))
    for _ in range(steps):
        y = torch.einsum("cij,cj->ci", K.expand(n ** dim, -1, -1), u[nodes])
        u = lay.solve(_zero_boundary(grid, grid.scatter(y) + rhs_f))
    return grid.give(u)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        state_rng = np.random.default_rng(seed + 1)
        for i, w in enumerate(_instances(case, seed)):
            if case["steps"]:
                L, n0, n = hierarchy_shape(w["n"])
                u0 = _bump(mesh.dof_coords(_hierarchy(2, 2, n0, L)[0][-1]), state_rng)
                out.append(_exact_steps(2, 2, n, w["eps"], 0.0, u0, case["steps"]) if i < 3 else None)
            elif dofs(2, w["order"], w["n"]) <= 17000:
                p = dict(eps=w["eps"], b=w["b"], f=1.0, c=0.0, delta0=1.0)
                out.append(_exact_stationary(2, w["order"], w["n"], p, True, w["order"])[1])
            else:
                out.append(None)
        return out
    dim, order, n = case["dim"], case["order"], _cells(case)
    if kind == "solve":
        rhs, sol = _exact_stationary(dim, order, n, _problem(case, seed), case["supg"], 1)
        return {"rhs": rhs, "sol": sol}
    if kind == "tcd":
        rng = np.random.default_rng(seed)
        eps, f = 10.0 ** rng.uniform(-4, -2), rng.uniform(0.0, 0.5)
        u0 = _bump(mesh.dof_coords(_hierarchy(dim, order, case["n0"], case["levels"])[0][-1]), rng)
        return _exact_steps(dim, order, n, eps, f, u0, 1)
    # one product, in slices of cells
    grid = _Grid(dim, order, n)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.rand(grid.m ** dim, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    lattice = _zero_boundary(grid, grid.take(x.cpu().numpy()))
    nodes = torch.as_tensor(grid.nodes, device=_device())
    ys, fs = [], []
    step = 2048
    for lo in range(0, n ** dim, step):
        part = np.arange(lo, min(lo + step, n ** dim))
        V = grid.vertices(part)
        forms = _Forms(dim, order, _warp(V) if case.get("warp") else V)
        if kind == "product":
            k, supg, degree = _constant(_problem(case, seed), forms), False, 1
        else:
            k = torch.tensor(_table(forms.x.cpu().numpy(), seed), device=_device())
            supg, degree = case["supg"], order
        y, F = forms.products(k, supg, degree, 1.0, lattice[nodes[part]])
        ys.append(y)
        fs.append(F)
    y = grid.scatter(torch.cat(ys))
    edge = torch.as_tensor(grid.output_order[grid.n_active:], device=y.device)
    y[edge] = lattice[edge]  # boundary rows are identity rows
    out = {"y": grid.give(y)}
    if kind == "assemble":
        out["rhs"] = grid.give(_zero_boundary(grid, grid.scatter(torch.cat(fs))))
    return out
