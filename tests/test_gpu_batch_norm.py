"""The norm of a batched Arnoldi vector where the second orthogonalisation removes most of it."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Batch, Context, TSystemCD2D, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smoother", [1, 3])
def test_exhausted_krylov_space(smoother):
    """9 inner unknowns and 30 iterations without a stop: from the tenth vector on what is left of w
    is rounding, and h2 is as large as w.  ||w||^2 - ||h2||^2 rounds to zero there, the norm of
    w - V h2 does not, so the residual estimate (a product of the rotations' sines) stays positive."""
    spaces, parents = mesh.structured_hierarchy(2, 1, 2, 2)
    co = coeffs(eps=0.1, b=(0.8, 0.6), f=1.0)
    B = Batch(solver_params(smoother=smoother, omega=0.8, stop_rule=1, red_factor=0.0, res_norm_min=0.0, maxit=30),
              Context())
    slot = B.submit(B.add_structure(spaces, parents), co, SUPG)
    B.run()
    x, info = B.fetch(slot, spaces[-1]["n_dof"])
    S = TSystemCD2D(spaces, parents, disctype=SUPG, coarse_disctype=SUPG)
    S.Init(co)
    want, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(want, rhs)
    S.Solve(want, rhs, solver_params(precision=0, stop_rule=1, red_factor=1e-13))
    assert info.iterations == 30 and 0.0 < info.final_residual < 1e-30
    assert np.linalg.norm(x - want) <= 1e-12 * np.linalg.norm(want)
