"""Solves whose finest matrix is streamed with bulk copies (4 M nonzeros and more, no matrix-free form)."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, TSystemCD2D, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 0])
def test_first_solve_tunes_the_product(precision):
    """The variant of the streamed product is chosen at the first solve, mixed or FP64."""
    spaces, parents = mesh.structured_hierarchy(2, 2, 5, 7)  # 320^2 cells, 6.5 M nonzeros
    S = TSystemCD2D(spaces, parents, disctype=SUPG)
    S.Init(coeffs(0, eps=1e-2, b=(0.8, 0.6), f=1.0, poly_degree=2))
    x, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(x, rhs)
    assert "not tuned yet" in S.ctx.product_tuning(S.sids[-1])
    info = S.Solve(x, rhs, solver_params(precision=precision, stop_rule=1, red_factor=1e-10, maxit=300))
    assert info.status == 0
    assert S.ctx.product_tuning(S.sids[-1]).startswith("chosen:")
    r0, r = np.linalg.norm(rhs), np.linalg.norm(rhs - S.ctx.spmv(S.sids[-1], x))
    assert r <= 1e-9 * r0
