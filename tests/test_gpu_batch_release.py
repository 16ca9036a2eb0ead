"""A time-dependent instance released between two steps leaves the grouped launches: the others step
on bit for bit as in a batch that never held it (its memory is returned to the pool at the
release, and the row kernels load an item's matrix before they look at its state)."""
import numpy as np
import pytest

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.system import Batch, CdgpuError, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu
TAU, THETA = 1e-3, (0.5, 0.5, 0.5, 0.5)


@pytest.mark.parametrize("smoother,omega", [(1, 0.8), (3, 1.0)])
def test_release_between_steps(smoother, omega):
    spaces, parents = mesh.structured_hierarchy(2, 2, 2, 5)
    n, na = int(spaces[-1]["n_dof"]), int(spaces[-1]["n_active"])
    prm = solver_params(smoother=smoother, omega=omega, stop_rule=1, red_factor=1e-10, restart=30, maxit=300)

    def states(keep, released):
        ctx = Context(0)
        try:
            B = Batch(prm, ctx)
            sid = B.add_structure(spaces, parents)
            with pytest.raises(CdgpuError):
                B.tcd_step(4)
            slots = {}
            for k in sorted(keep + released):
                u0 = np.random.default_rng(k).standard_normal(n)
                u0[na:] = 0.0
                slots[k] = B.submit_tcd(sid, coeffs(_lib.COEFF_ROTATING, eps=10.0 ** -(2 + k), f=0.1 * k), TAU, *THETA, u0)
            B.tcd_step(4)
            for k in released:
                B.release(slots[k])
            for _ in range(2):
                B.tcd_step(4)
            out = [B.fetch(slots[k], n)[0] for k in keep]
            for k in keep:
                B.release(slots[k])
            B.tcd_step(4)  # nothing left: nothing to do
            return out
        finally:
            ctx.close()

    for a, b in zip(states([0, 2], [1, 3]), states([0, 2], [])):
        assert np.isfinite(a).all() and np.array_equal(a, b)
