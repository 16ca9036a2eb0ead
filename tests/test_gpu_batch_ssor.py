"""The batched cycle's SSOR sweeps, where two passes meeting in one colour class are made as one,
against plain passes in numpy: after one FGMRES iteration the solution is a multiple of the cycle's
result, so the whole V-cycle (the finest level in grouped launches, the ones below in one block)
shows in it.  omega away from 1, where the second update of a class is not void; 1 to 3 sweeps."""
import numpy as np
import pytest
import scipy.sparse as sps

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Batch, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu


def _points(sp):
    """coordinates of the (bi)linear unknowns: local unknown k of a cell is its corner k in
    lexicographic order"""
    d, nv = sp["dim"], 2 ** sp["dim"]
    X = np.asarray(sp["coords"]).reshape(-1, nv, d)
    gn = np.asarray(sp["global_numbers"]).reshape(-1, nv)
    lo, hi = X.min(1), X.max(1)
    P = np.zeros((sp["n_dof"], d))
    for k in range(nv):
        P[gn[:, k]] = np.stack([(hi if k >> q & 1 else lo)[:, q] for q in range(d)], 1)
    return P


def _prolongation(fine, coarse, n):
    pf, pc = _points(fine), _points(coarse)
    W = np.ones((len(pf), len(pc)))
    for q in range(pf.shape[1]):
        W *= np.maximum(0.0, 1.0 - n * np.abs(pf[:, q, None] - pc[None, :, q]))
    W[fine["n_active"]:] = 0.0
    W[:, coarse["n_active"]:] = 0.0
    return W


def _classes(rp, kc, na):
    col = np.full(na, -1)
    for r in range(na):
        used = {col[c] for c in kc[rp[r]:rp[r + 1]] if c < na and c != r}
        col[r] = next(c for c in range(na) if c not in used)
    return [np.flatnonzero(col == c) for c in range(col.max() + 1)]


def _sweeps(A, cls, x, f, omega, count):
    d = np.diag(A)
    for _ in range(count):
        for rows in cls + cls[::-1]:
            x[rows] += omega * (f[rows] - A[rows] @ x) / d[rows]
    return x


def _cycle(lev, l, f, omega, pre, post):
    A, cls, P = lev[l]
    if l == 0:
        return np.linalg.solve(A, f)
    x = _sweeps(A, cls, np.zeros_like(f), f, omega, pre)
    x += P @ _cycle(lev, l - 1, P.T @ (f - A @ x), omega, pre, post)
    return _sweeps(A, cls, x, f, omega, post)


@pytest.mark.parametrize("dim,n0,levels,omega,pre,post", [
    (2, 3, 3, 0.7, 2, 2), (2, 5, 2, 1.3, 1, 1), (2, 2, 4, 1.2, 3, 2), (3, 2, 3, 0.8, 2, 1)])
def test_cycle_of_ssor_sweeps(dim, n0, levels, omega, pre, post):
    spaces, parents = mesh.structured_hierarchy(dim, 1, n0, levels)
    co = coeffs(0, eps=5e-2, b=(0.8, 0.6, 0.3)[:dim], f=1.0, poly_degree=1)
    ctx = Context(0)
    try:
        B = Batch(solver_params(smoother=3, omega=omega, pre=pre, post=post, maxit=1, red_factor=0.0,
                                restart=10), ctx)
        slot = B.submit(B.add_structure(spaces, parents), co, SUPG)
        B.run(1)
        n, na = spaces[-1]["n_dof"], spaces[-1]["n_active"]
        x, info = B.fetch(slot, n)
        assert info.iterations == 1
        lev = []
        for l, sp in enumerate(spaces):
            sid = ctx.upload_space(sp)
            nnz = ctx.build_pattern(sid)
            ctx.set_coeffs(sid, co)
            ent, rhs = ctx.assemble(sid, SUPG, sp["n_dof"], nnz)
            rp, kc = ctx.get_pattern(sid, sp["n_dof"], nnz)
            a = sp["n_active"]
            A = sps.csr_matrix((ent, kc, rp), shape=(sp["n_dof"],) * 2).toarray()[:a, :a]
            P = _prolongation(sp, spaces[l - 1], n0 << (l - 1))[:a, :spaces[l - 1]["n_active"]] if l else None
            lev.append((A, _classes(rp, kc, a), P))
        f = rhs[:na]
        z = _cycle(lev, levels - 1, f, omega, pre, post)
        Az = lev[-1][0] @ z
        want = (Az @ f) / (Az @ Az) * z
        # the cycle runs in FP32: at most about 66 classes of 12 roundings each on every level
        tol = levels * 66 * 12 * 6e-8
        assert np.linalg.norm(x[:na] - want) <= tol * np.linalg.norm(want)
    finally:
        ctx.close()
