"""One hierarchy of 32^3 triquadratic cells (15.8 M nonzeros) through the forms its finest operator
takes: matrix-free with 10 (Galerkin) and 13 (SUPG) tensors, and, with tabulated coefficients, the
streamed matrix (FP64 sweeps, defect and last sweep by bulk copies inside the captured cycle) or the
FP32 CSR kernels.  Each re-assembly changes the form, so the captured cycles are made again; every
cycle is compared with the one written in numpy (test_gpu_dense_cycle.py) on the assembled entries.

Tolerances as there: 1e-11 in FP64; mixed 2e-4 with FP32 CSR levels, 5e-3 with tensor-core products
(TF32 inputs)."""
import numpy as np
import pytest
import scipy.sparse as sps

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.system import GALERKIN, SUPG, Context, TSystemCD3D, coeffs, solver_params
from test_gpu_dense_cycle import cycle

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
B3 = (0.6, 0.64, 0.48)


def _table(xyz):
    x, y, z = xyz[..., 0], xyz[..., 1], xyz[..., 2]
    out = np.zeros(xyz.shape[:-1] + (6,))
    out[..., 0] = 2e-2 * (1.0 + 0.5 * np.sin(3.0 * x + y))
    out[..., 1], out[..., 2], out[..., 3] = 0.5 - y, x - 0.5, 0.2 * np.cos(2.0 * z)
    out[..., 4], out[..., 5] = 0.1, 1.0 + z
    return out


@pytest.fixture(scope="module")
def problem(oracle_lib):
    spaces, parents = mesh.structured_hierarchy(3, 2, 2, 5)
    ctx = Context(0)
    sids, levels = [], []
    for l, sp in enumerate(spaces):
        sid = ctx.upload_space(sp)
        nnz = ctx.build_pattern(sid)
        lv = dict(na=sp["n_active"], pat=ctx.get_pattern(sid, sp["n_dof"], nnz), nnz=nnz)
        if l > 0:
            r, c, v = oracle_lib.prolongation(3, 2, spaces[l - 1], dict(sp), parents[l])
            lv["P"] = sps.csr_matrix((v, c, r), shape=(sp["n_dof"], spaces[l - 1]["n_dof"]))
        sids.append(sid)
        levels.append(lv)
    yield ctx, spaces, sids, ctx.hierarchy(sids, parents), levels
    ctx.close()


def test_reassembly_changes_the_form(problem):
    ctx, spaces, sids, mg, levels = problem
    n, na = spaces[-1]["n_dof"], spaces[-1]["n_active"]
    rng = np.random.default_rng(8)
    for form in ("galerkin", "supg", "table", "galerkin", "table", "supg"):
        disc = SUPG if form == "supg" else GALERKIN
        for sp, sid, lv in zip(spaces, sids, levels):
            if form == "table":
                ctx.set_coeffs(sid, coeffs(_lib.COEFF_TABLE), _table(ctx.quadrature_points(sid, sp["n_cells"], 3)))
            else:
                ctx.set_coeffs(sid, coeffs(0, eps=1e-2, b=B3, c=0.3, f=1.0))
            ent, _ = ctx.assemble(sid, disc, sp["n_dof"], lv["nnz"])
            rp, kc = lv["pat"]
            lv["A"] = sps.csr_matrix((ent, kc, rp), shape=(sp["n_dof"],) * 2)
            lv["d"] = lv["A"].diagonal()
        f = rng.standard_normal(n)
        start = f.copy()
        start[:na] = 0.0
        ref = cycle(levels, 4, f, start, 2, 2, 0.8, 1.0, 1)
        for precision, tol in ((0, 1e-11), (1, 2e-4 if form == "table" else 5e-3)):
            prm = solver_params(solver=11, precision=precision, maxit=1, red_factor=0.0, div_factor=1e30)
            x, _ = ctx.solve(mg, prm, f, np.zeros(n))
            err = np.abs(x - ref).max() / np.abs(ref).max()
            print(f"{form} precision {precision}: {err:.2e}")
            assert err <= tol, (form, precision)
        # the streamed product as the solve tuned it: rows of at most 125 terms
        assert ctx.product_tuning(sids[-1]).startswith("chosen:")
        A = levels[-1]["A"]
        assert np.all(np.abs(ctx.spmv(sids[-1], f) - A @ f) <= 130 * EPS * (abs(A) @ np.abs(f)))


@pytest.mark.parametrize("precision", [0, 1])
def test_supg_solve_against_the_matrix(precision):
    """The solves that apply the SUPG operator without the matrix, by the residual of their solution
    with the assembled entries: below 1e-12 by the recurrence, and off it by the two products'
    rounding (some 1e-15 ||A|| ||x||, and ||A|| ||x|| / ||f|| is below 1e3), 1e-11."""
    spaces, parents = mesh.structured_hierarchy(3, 2, 2, 5)
    S = TSystemCD3D(spaces, parents, disctype=SUPG, coarse_disctype=SUPG)
    S.Init(coeffs(0, eps=1e-2, b=B3, c=0.1, f=1.0, delta0=1.0 / 3.0))
    x, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(x, rhs)
    info = S.Solve(x, rhs, solver_params(precision=precision, stop_rule=1, red_factor=1e-12))
    assert info.status == 0
    sid, sp = S.sids[-1], spaces[-1]
    nnz = S.ctx.build_pattern(sid)
    rp, kc = S.ctx.get_pattern(sid, sp["n_dof"], nnz)
    ent, f = S.ctx.assemble(sid, SUPG, sp["n_dof"], nnz)
    A = sps.csr_matrix((ent, kc, rp), shape=(sp["n_dof"],) * 2)
    assert np.linalg.norm(f - A @ x) <= 1e-11 * np.linalg.norm(f)
