"""One theta step's matrix work in one pass over the entries: the system matrix, the mass matrix
it leaves and the right-hand side against the separate updates in numpy, on levels smaller than
a block, rows longer than one turn of a row's lanes, and both rules for the coarse levels."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import Context, TSystemTCD2D, TSystemTCD3D, coeffs, solver_params

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _pattern(space):
    ctx = Context(0)
    try:
        sid = ctx.upload_space(space)
        return ctx.get_pattern(sid, space["n_dof"], ctx.build_pattern(sid))
    finally:
        ctx.close()


@pytest.mark.parametrize("dim,order,n0,levels", [(2, 1, 2, 1), (2, 1, 3, 4), (2, 2, 5, 2), (3, 1, 2, 3), (3, 2, 2, 2)])
def test_step_matrices(dim, order, n0, levels):
    tau, th = 0.04, (0.3, 0.7, 0.6, 0.4)
    spaces, parents = mesh.structured_hierarchy(dim, order, n0, levels)
    ctx = Context(0)
    try:
        S = (TSystemTCD2D if dim == 2 else TSystemTCD3D)(spaces, parents, ctx=ctx)
        S.Init(coeffs(0, eps=0.05, b=(1.0, 0.5, 0.25)[:dim], c=0.1, f=1.0))
        n, na = spaces[-1]["n_dof"], spaces[-1]["n_active"]
        rng = np.random.default_rng(5)
        sol = rng.standard_normal(n)
        S.AssembleMRhs(sol)  # also sets the Dirichlet entries
        u0 = sol.copy()
        f_old = S.rhs()
        for sid in S.sids:
            ctx.set_coeffs(sid, coeffs(0, eps=0.05, b=(1.0, 0.5, 0.25)[:dim], c=0.1, f=1.7))
        S.AssembleARhs()
        f = S.rhs()
        pats = [_pattern(s) for s in spaces]
        before = [S.matrices(l, len(pats[l][1]))[:2] for l in range(levels)]
        info = S.Step(sol, tau, *th, params=solver_params(red_factor=1e-12, restart=32, maxit=200))
        assert info.status == 0
        for l in range(levels):
            rp, kc = pats[l]
            M0, A = before[l]
            M1, A1, Sy = S.matrices(l, len(kc))
            half = dim == 2 or l == levels - 1
            ka = int(rp[spaces[l]["n_active"]])
            K = M0 - tau * th[1] * A if half else M0.copy()
            want = K + (tau * th[1] + tau * th[0]) * A if half else K + tau * th[0] * A
            # three updates of one rounding each here, two roundings each in numpy
            tol = 8 * EPS * (np.abs(M0) + tau * (th[0] + 2 * th[1]) * np.abs(A))
            assert np.all(np.abs(Sy - want)[:ka] <= tol[:ka])
            assert np.all(np.abs(M1 - (want - tau * th[0] * A))[:ka] <= tol[:ka])
            assert np.array_equal(Sy[ka:], M0[ka:]) and np.array_equal(M1[ka:], M0[ka:])
            assert np.array_equal(A1, A)
        rows = np.repeat(np.arange(n), np.diff(rp))
        mul = lambda v, x: np.bincount(rows, v * x[kc], n)
        B = tau * th[2] * f_old + tau * th[3] * f + mul(K, u0)
        start = np.concatenate([u0[:na], f[na:]])
        assert np.array_equal(sol[na:], f[na:])
        r0, r = (B - mul(Sy, start))[:na], (B - mul(Sy, sol))[:na]
        # the solve stops at 1e-12 of its first residual; the rest is the rounding of B and of
        # the residuals, at most the row length + 4 roundings per row
        length = np.diff(rp).max() + 4
        rounding = EPS * length * (np.abs(B) + mul(np.abs(K), np.abs(u0)) + 2 * mul(np.abs(Sy), np.abs(sol)))[:na]
        assert np.linalg.norm(r) <= 1.01e-12 * np.linalg.norm(r0) + 4 * np.linalg.norm(rounding)
    finally:
        ctx.close()
