"""Batched Jacobi sweeps with damping 0: the start of a coarse level's sweeps is zero in both of its
vectors, not what an earlier cycle left there."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Batch, Context, TSystemCD2D, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2)])
def test_zero_damping(pre, post):
    """8 iterations, below the coarse-space correction's stagnation, on levels of 3,969, 961 and 225
    inner unknowns (the last of them and below in one block): the same as the single mixed solve.
    Cycles in FP32 differ by their rounding, 2^-24 times the cycle's condition, and the iterates by
    the Krylov coefficients' share of it; a stale coarse vector is an error of the size of x."""
    spaces, parents = mesh.structured_hierarchy(2, 1, 4, 5)
    co = coeffs(eps=0.1, b=(0.8, 0.6), f=1.0)
    prm = dict(smoother=1, omega=0.0, pre=pre, post=post, stop_rule=1, red_factor=1e-14, maxit=8)
    B = Batch(solver_params(**prm), Context())
    slot = B.submit(B.add_structure(spaces, parents), co, SUPG)
    B.run()
    x, info = B.fetch(slot, spaces[-1]["n_dof"])
    S = TSystemCD2D(spaces, parents, disctype=SUPG, coarse_disctype=SUPG)
    S.Init(co)
    want, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(want, rhs)
    S.Solve(want, rhs, solver_params(precision=1, **prm))
    assert np.linalg.norm(x - want) <= 1e-3 * np.linalg.norm(want)
