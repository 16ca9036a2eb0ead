"""The inverse of the coarsest active block by one warp (at most 32 rows) and by one block (more):
with one level the cycle is the exact solve, so FGMRES stops after its first iteration and the
solution is that of a direct solve of the assembled matrix.  Sizes from one row to both sides of
the limit (25, 27 | 36 and 49 rows); a convection-dominated Galerkin matrix, whose elimination
interchanges rows, and a diffusive one.  The batch inverts by the same kernels."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import GALERKIN, Batch, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1.0, 1e-3])
@pytest.mark.parametrize("dim,order,n0", [(2, 1, 2), (2, 1, 4), (2, 2, 3), (3, 2, 2), (2, 1, 7), (2, 2, 4)])
def test_one_level_solve(dim, order, n0, eps):
    spaces, parents = mesh.structured_hierarchy(dim, order, n0, 1)
    sp = spaces[0]
    n, na = sp["n_dof"], sp["n_active"]
    co = coeffs(0, eps=eps, b=(0.8, 0.6, 0.3)[:dim], f=1.0, poly_degree=order)
    ctx = Context(0)
    try:
        sid = ctx.upload_space(sp)
        nnz = ctx.build_pattern(sid)
        ctx.set_coeffs(sid, co)
        ent, rhs = ctx.assemble(sid, GALERKIN, n, nnz)
        rp, kc = ctx.get_pattern(sid, n, nnz)
        A = np.zeros((n, n))
        A[np.repeat(np.arange(n), np.diff(rp)), kc] = ent
        A = A[:na, :na]
        want = np.linalg.solve(A, rhs[:na])
        # both sides eliminate with partial pivoting: n roundings per entry, amplified by the
        # condition; the stopping test leaves 1e-10 of the right-hand side before the first iteration only
        tol = 8 * na * np.finfo(float).eps * np.linalg.cond(A)
        assert tol < 1e-6
        x, info = ctx.solve(ctx.hierarchy([sid], parents), solver_params(red_factor=1e-10), rhs, np.zeros(n))
        assert info.status == 0 and info.iterations == 1
        assert np.abs(x[:na] - want).max() <= tol * np.abs(want).max()
        B = Batch(solver_params(red_factor=1e-10), ctx)
        slot = B.submit(B.add_structure(spaces, parents), co, GALERKIN)
        B.run(2)
        y, info = B.fetch(slot, n)
        # (its preconditioner hands the result over in 32 bits: a second iteration or a third)
        assert info.status == 0 and info.iterations <= 3
        res = np.linalg.norm(rhs[:na] - A @ y[:na])
        assert res <= 1.01e-10 * np.linalg.norm(rhs[:na])
    finally:
        ctx.close()
