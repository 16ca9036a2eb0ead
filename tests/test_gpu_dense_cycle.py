"""The coarse levels' V-cycle applied as one dense matrix (coarse.cuh), against the cycle itself.

One fixed-point iteration from a zero start returns x = M^-1 f, one multigrid cycle of f.  It is
compared with TMultiGrid3D::Cycle (src/FE/MultiGrid3D.C:423-669) written in numpy on the
library's own matrices and the oracle's transfers: damped Jacobi sweeps on every level, exact
solve at the bottom.  FP64: the two differ by the rounding of a few hundred operations per entry
on matrices whose coarse inverses have condition numbers below 1e4, so 1e-11 relative; the mixed
form runs the finer levels in FP32, 2e-4.

The dense level is the last one of at most 1,024 active rows below the finest.  Cases: no coarse
level small enough but the bottom; the bottom with no active row (one Q1 cell); every mix of
sweep counts (the iterates alternate between two buffers, the first sweep has no matrix); long
rows (3D Q2); 961 rows (eight columns per block, a partly filled last block); 729 rows in 3D; a
W-cycle and an iterative coarse smoother, which keep the cycle as it was.
"""
import numpy as np
import pytest
import scipy.sparse as sps
import scipy.sparse.linalg as spl

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import GALERKIN, SUPG, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from parmoon_cmg_b200 import _build
    _build.build()
    c = Context(0)
    yield c
    c.close()


def hierarchy(ctx, oracle_lib, dim, order, n0, L, disc=SUPG):
    co = coeffs(0, eps=1e-2, b=(0.8, 0.6) if dim == 2 else (0.6, 0.64, 0.48), c=0.3, f=1.0)
    spaces, parents = mesh.structured_hierarchy(dim, order, n0, L)
    levels, sids = [], []
    for l, sp in enumerate(spaces):
        sid = ctx.upload_space(sp)
        nnz = ctx.build_pattern(sid)
        ctx.set_coeffs(sid, co)
        ent, _ = ctx.assemble(sid, disc, sp["n_dof"], nnz)
        rp, kc = ctx.get_pattern(sid, sp["n_dof"], nnz)
        lv = dict(A=sps.csr_matrix((ent, kc, rp), shape=(sp["n_dof"],) * 2), na=sp["n_active"])
        lv["d"] = lv["A"].diagonal()
        if l > 0:
            r, c, v = oracle_lib.prolongation(dim, order, spaces[l - 1], dict(sp), parents[l])
            lv["P"] = sps.csr_matrix((v, c, r), shape=(sp["n_dof"], spaces[l - 1]["n_dof"]))
        levels.append(lv)
        sids.append(sid)
    return sids, parents, levels


def cycle(levels, l, f, start, pre, post, omega, damp, recursions):
    """the cycle on level l from `start` (Dirichlet entries of f, else zero, at the top)"""
    lv = levels[l]
    na, A, d = lv["na"], lv["A"], lv["d"]
    if l == 0:
        x = f.copy()
        if na:
            x[:na] = spl.spsolve(sps.csc_matrix(A[:na, :na]), f[:na] - A[:na, na:] @ f[na:])
        return x

    def sweep(x):
        y = x + omega * (f - A @ x) / d
        y[na:] = f[na:]
        return y
    x = start.copy()
    for _ in range(pre):
        x = sweep(x)
    nac = levels[l - 1]["na"]
    fc = lv["P"].T @ (f - A @ x)
    fc[nac:] = 0.0
    xc = np.zeros_like(fc)
    for _ in range(recursions if l > 1 else 1):
        xc = cycle(levels, l - 1, fc, xc, pre, post, omega, damp, recursions)
    x[:na] += damp * (lv["P"] @ xc)[:na]
    for _ in range(post):
        x = sweep(x)
    return x


@pytest.mark.parametrize("dim,order,n0,L,pre,post,omega,damp,w", [
    (2, 1, 1, 6, 2, 2, 0.8, 1.0, 1),
    (2, 1, 4, 5, 1, 0, 0.8, 1.0, 1),
    (2, 1, 4, 5, 0, 1, 0.7, 1.0, 1),
    (2, 1, 2, 6, 3, 2, 0.8, 0.9, 1),
    (2, 1, 17, 3, 2, 2, 0.8, 1.0, 1),
    (2, 2, 3, 4, 2, 1, 0.8, 1.0, 1),
    (2, 2, 2, 5, 1, 3, 0.6, 1.1, 1),
    (3, 1, 5, 3, 2, 2, 0.8, 1.0, 1),
    (3, 2, 2, 3, 2, 2, 0.8, 1.0, 1),
    (3, 2, 1, 4, 4, 1, 0.5, 1.0, 1),
    (2, 2, 2, 4, 2, 2, 0.8, 1.0, 2),
])
def test_one_cycle(ctx, oracle_lib, dim, order, n0, L, pre, post, omega, damp, w):
    sids, parents, levels = hierarchy(ctx, oracle_lib, dim, order, n0, L)
    mg = ctx.hierarchy(sids, parents)
    n, na = levels[-1]["A"].shape[0], levels[-1]["na"]
    rng = np.random.default_rng(pre * 100 + post * 10 + dim)
    for precision, tol in ((0, 1e-11), (1, 2e-4)):
        f = rng.standard_normal(n)
        start = f.copy()
        start[:na] = 0.0
        ref = cycle(levels, L - 1, f, start, pre, post, omega, damp, w)
        prm = solver_params(solver=11, precision=precision, pre=pre, post=post, omega=omega, gmg_damp=damp, cycle=w,
                            maxit=1, red_factor=0.0, res_norm_min=0.0, div_factor=1e30)
        x, info = ctx.solve(mg, prm, f, np.zeros(n))
        err = np.abs(x - ref).max() / np.abs(ref).max()
        print(f"precision {precision}: {err:.2e}")
        assert err <= tol


@pytest.mark.parametrize("disc", [GALERKIN, SUPG])
def test_one_cycle_with_matrix_free_sweeps(ctx, oracle_lib, disc):
    """32^3 Q2 cells: the finest level's sweeps and defect are applied without the matrix in both
    forms (10 and 13 tensors), the coarse levels as above.  The mixed form's tensor-core products
    round their inputs to TF32 (2^-11 relative), 5e-3."""
    sids, parents, levels = hierarchy(ctx, oracle_lib, 3, 2, 2, 5, disc)
    mg = ctx.hierarchy(sids, parents)
    n, na = levels[-1]["A"].shape[0], levels[-1]["na"]
    f = np.random.default_rng(disc).standard_normal(n)
    start = f.copy()
    start[:na] = 0.0
    ref = cycle(levels, 4, f, start, 2, 2, 0.8, 1.0, 1)
    for precision, tol in ((0, 1e-11), (1, 5e-3)):
        prm = solver_params(solver=11, precision=precision, maxit=1, red_factor=0.0, div_factor=1e30)
        x, info = ctx.solve(mg, prm, f, np.zeros(n))
        err = np.abs(x - ref).max() / np.abs(ref).max()
        print(f"disc {disc} precision {precision}: {err:.2e}")
        assert err <= tol


def test_follows_assembly_and_parameters(ctx, oracle_lib):
    """The matrix is formed again when the coefficients, the sweeps or the damping change between
    solves of one hierarchy, and left when they do not."""
    sids, parents, levels = hierarchy(ctx, oracle_lib, 2, 1, 4, 5)
    mg = ctx.hierarchy(sids, parents)
    n = levels[-1]["A"].shape[0]
    f = np.random.default_rng(3).standard_normal(n)
    f[levels[-1]["na"]:] = 0.0

    def solve(**kw):
        return ctx.solve(mg, solver_params(solver=11, maxit=1, red_factor=0.0, **kw), f, np.zeros(n))[0]
    a = solve(pre=2)
    b = solve(pre=1)
    assert np.array_equal(solve(pre=2), a) and not np.array_equal(a, b)
    assert not np.array_equal(solve(pre=2, omega=0.5), a)
    for sid in sids:
        ctx.set_coeffs(sid, coeffs(0, eps=0.1, b=(0.0, 1.0), c=0.0, f=1.0))
    ctx.assemble_hierarchy(mg, SUPG)
    c = solve(pre=2)
    fresh, sids2 = Context(0), []
    spaces, par2 = mesh.structured_hierarchy(2, 1, 4, 5)
    for sp in spaces:
        sid = fresh.upload_space(sp)
        fresh.build_pattern(sid)
        fresh.set_coeffs(sid, coeffs(0, eps=0.1, b=(0.0, 1.0), c=0.0, f=1.0))
        sids2.append(sid)
    mg2 = fresh.hierarchy(sids2, par2)
    fresh.assemble_hierarchy(mg2, SUPG)
    d = fresh.solve(mg2, solver_params(solver=11, maxit=1, red_factor=0.0, pre=2), f, np.zeros(n))[0]
    fresh.close()
    assert np.array_equal(c, d) and not np.array_equal(c, a)
