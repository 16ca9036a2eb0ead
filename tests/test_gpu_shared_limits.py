"""Coarse cycles in shared memory at its limit: many levels of one mesh (identity transfers)."""
import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import SUPG, Batch, Context, TSystemCD2D, coeffs, solver_params

pytestmark = pytest.mark.gpu
CO = dict(eps=0.1, b=(0.8, 0.6), f=1.0)


def _levels(n):
    """n levels of the 32^2 bilinear mesh, 961 inner unknowns each."""
    sp = mesh.structured_hierarchy(2, 1, 32, 1)[0][0]
    return [sp] * n, [None] + [np.arange(sp["n_cells"], dtype=np.int32)] * (n - 1)


def _solution(spaces, parents, **prm):
    S = TSystemCD2D(spaces, parents, disctype=SUPG, coarse_disctype=SUPG)
    S.Init(coeffs(**CO))
    x, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(x, rhs)
    info = S.Solve(x, rhs, solver_params(stop_rule=1, red_factor=1e-12, **prm))
    assert info.status == 0
    return x


@pytest.mark.parametrize("levels", [8, 9, 14])
def test_dense_cycle_at_the_limit(levels):
    """The vectors of seven levels above the coarsest fit beside each other, 227 KB, but for their
    flags: the dense level is one below.  (14: as many levels as there may be, and more.)"""
    x = _solution(*_levels(levels))
    want = _solution(*_levels(2))
    assert np.linalg.norm(x - want) <= 1e-9 * np.linalg.norm(want)


def test_batches_with_different_needs():
    """A second batch whose coarse levels need less shared memory (60 KB) leaves what the first one
    captures again afterwards (93 KB, another number of iterations per graph) its own."""
    prm = solver_params(smoother=3, omega=1.0, pre=1, post=1, stop_rule=1, red_factor=1e-11, maxit=100)
    sp = _levels(1)[0][0]
    u0 = np.exp(-((mesh.dof_coords(sp) - 0.35) ** 2).sum(1) / (2 * 0.1 ** 2))
    u0[sp["n_active"]:] = 0.0

    def first_step(ctx, n):
        B = Batch(prm, ctx)
        slot = B.submit_tcd(B.add_structure(*_levels(n)), coeffs(**CO), 1e-2, 0.5, 0.5, 0.5, 0.5, u0)
        B.tcd_step(4)
        return B, slot

    ctx = Context()
    A, slot = first_step(ctx, 12)
    first_step(ctx, 8)
    A.tcd_step(5)
    W, wslot = first_step(Context(), 2)
    W.tcd_step(5)
    x, want = A.fetch(slot, sp["n_dof"])[0], W.fetch(wslot, sp["n_dof"])[0]
    assert np.linalg.norm(x - want) <= 1e-8 * np.linalg.norm(want)
