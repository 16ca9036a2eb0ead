"""The batched cycle's split of the levels: grouped launches above, one block below (b_cta_cycle).

With damped Jacobi an instance runs the algorithm of the mixed single solve, whose cycle is checked
against the reference's on its own: same stopping rule, the same solution up to the stopping
residual (1e-12 of ||f|| times a condition number below 1e3: 1e-9), iterations within one.  SOR and
SSOR are checked against a direct solve of the assembled matrix (1e-8).  Shapes: one level; the
bottom alone below the finest; active rows on both sides of the one-block limits (225 | 961 for
Jacobi, 961 | 1,089 for SOR and SSOR); hexahedra of both orders; all of them in one batch, so that
the launches of a depth serve some of the instances only.
"""
import numpy as np
import pytest
import scipy.sparse as sps
import scipy.sparse.linalg as spl

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Batch, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu

SHAPES = [  # dim, order, n0, levels
    (2, 1, 9, 1), (2, 2, 6, 2), (2, 1, 4, 4), (2, 1, 8, 4), (2, 1, 17, 3), (2, 2, 2, 6), (2, 2, 17, 2), (2, 1, 1, 5),
    (3, 1, 5, 3), (3, 2, 2, 3),
]


@pytest.fixture(scope="module")
def ctx():
    from parmoon_cmg_b200 import _build
    _build.build()
    c = Context(0)
    yield c
    c.close()


def coefficients(dim, order):
    return coeffs(0, eps=3e-2, b=(0.8, 0.6) if dim == 2 else (0.6, 0.64, 0.48), f=1.0, poly_degree=order)


@pytest.mark.parametrize("smoother,pre,post", [(1, 2, 2), (1, 1, 2), (2, 2, 1), (3, 2, 2), (3, 1, 0)])
def test_levels_in_launches_and_in_one_block(ctx, smoother, pre, post):
    prm = solver_params(smoother=smoother, omega=0.8 if smoother == 1 else 1.0, pre=pre, post=post, stop_rule=1,
                        red_factor=1e-12, maxit=400)
    B = Batch(prm, ctx)
    slots = []
    for dim, order, n0, L in SHAPES:
        spaces, parents = mesh.structured_hierarchy(dim, order, n0, L)
        sid = B.add_structure(spaces, parents)
        slots.append((B.submit(sid, coefficients(dim, order), SUPG), spaces, parents, dim, order))
    B.run(5)
    for slot, spaces, parents, dim, order in slots:
        n = int(spaces[-1]["n_dof"])
        x, info = B.fetch(slot, n)
        assert info.status == 0, (dim, order, n, info.iterations)
        sids = []
        for sp in spaces:
            sid = ctx.upload_space(sp)
            nnz = ctx.build_pattern(sid)
            ctx.set_coeffs(sid, coefficients(dim, order))
            ent, rhs = ctx.assemble(sid, SUPG, sp["n_dof"], nnz)
            sids.append(sid)
        if smoother == 1:
            ref, one = ctx.solve(ctx.hierarchy(sids, parents), solver_params(
                precision=1, omega=0.8, pre=pre, post=post, stop_rule=1, red_factor=1e-12, maxit=400), rhs, np.zeros(n))
            tol = 1e-9
            assert abs(info.iterations - one.iterations) <= 1, (dim, order, n, info.iterations, one.iterations)
        else:
            rp, kc = ctx.get_pattern(sids[-1], n, len(ent))
            ref, tol = spl.spsolve(sps.csc_matrix(sps.csr_matrix((ent, kc, rp), shape=(n, n))), rhs), 1e-8
        err = np.abs(x - ref).max() / np.abs(ref).max()
        assert err <= tol, (dim, order, n, err)
