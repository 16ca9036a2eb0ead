"""The Gram-Schmidt kernels of FGMRES over every basis size of a restart cycle.

FGMRES reports |s_{i+1}|, the residual norm that follows from its own orthogonalisation
coefficients, when it stops on its residual test; with a correct Arnoldi relation V H = A Z it
equals ||f - A x|| of the solution it returns.  A wrong, missing or twice-counted block of rows in any of the sums breaks the relation
by a relative amount of about 1 / blocks.  A run that stops at iteration `its` has used the basis sizes
1 .. min(its, restart): the rows-per-thread steps (K < 8,
< 16, >= 16), the one-block-per-SM sizes (K > 24), the largest basis (32) and a restart.  The
estimate carries rounding of about its * 1e-16 * ||r0||, so with residuals above 1e-3 ||r0|| a
relative 1e-10 bounds it.
"""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from parmoon_cmg_b200 import _build
    _build.build()
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("dim,order,n0,levels,its,restart,red", [
    (2, 1, 4, 2, 7, 32, 0.13),     # 81 rows: one partly filled block
    (2, 1, 5, 4, 26, 32, 0.069),   # 1,681 rows
    (2, 2, 3, 6, 32, 32, 0.0412),  # 37,249 rows, the largest basis
    (2, 2, 4, 6, 27, 20, 0.0912),  # 66,049 rows, several rows per thread in one pass, a restart
    (3, 2, 2, 5, 9, 32, 0.0622),   # 274,625 rows: the matrix-free product's fused first pass
])
@pytest.mark.parametrize("precision", [0, 1])
def test_reported_residual_is_the_true_one(ctx, dim, order, n0, levels, its, restart, red, precision):
    spaces, parents = mesh.structured_hierarchy(dim, order, n0, levels)
    co = coeffs(0, eps=2e-3 if dim == 2 else 1e-2, b=(0.8, 0.6) if dim == 2 else (0.6, 0.64, 0.48), f=1.0)
    sids = []
    for sp in spaces:
        sid = ctx.upload_space(sp)
        ctx.build_pattern_device(sid)
        ctx.set_coeffs(sid, co)
        sids.append(sid)
    mg = ctx.hierarchy(sids, parents)
    ctx.assemble_hierarchy(mg, SUPG)
    n, na = int(spaces[-1]["n_dof"]), int(spaces[-1]["n_active"])
    rng = np.random.default_rng(its)
    rhs = rng.standard_normal(n)
    rhs[na:] = 0.0
    # a light smoother, so that `its` iterations leave a residual well above rounding
    prm = solver_params(precision=precision, pre=1, post=0, omega=0.05, restart=restart, maxit=100, stop_rule=1,
                        red_factor=red, res_norm_min=0.0)
    x, info = ctx.solve(mg, prm, rhs, np.zeros(n))
    d, res = ctx.defect(sids[-1], x, rhs)
    ratio = res / info.initial_residual
    print(f"n={n} its={info.iterations} ratio={ratio:.2e} estimate/true-1={info.final_residual / res - 1:.2e}")
    assert info.status == 0
    assert info.iterations >= min(its - 2, restart + 1)
    assert abs(info.initial_residual / np.linalg.norm(rhs) - 1) <= 1e-12 and ratio > 1e-3
    assert abs(info.final_residual / res - 1) <= 1e-10
