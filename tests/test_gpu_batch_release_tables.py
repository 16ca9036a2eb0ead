"""The tables of a batch are made again without a time-dependent instance that is released between
two steps: what its arrays held is not loaded any more.  Seen where the last one goes, after
which a step launches nothing (with the tables kept, the step's graph would run once more)."""
import numpy as np
import pytest

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.system import Batch, Context, coeffs, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3])
def test_step_after_the_last_release(count):
    spaces, parents = mesh.structured_hierarchy(2, 2, 2, 4)
    ctx = Context(0)
    try:
        B = Batch(solver_params(stop_rule=1, red_factor=1e-10, restart=30, maxit=300), ctx)
        sid = B.add_structure(spaces, parents)
        u0 = np.zeros(spaces[-1]["n_dof"])
        slots = [B.submit_tcd(sid, coeffs(_lib.COEFF_ROTATING, eps=1e-2, f=1.0 + k), 1e-3, 0.5, 0.5, 0.5, 0.5, u0)
                 for k in range(count)]
        assert B.tcd_step(4) > 0
        mode, graphs, host = B.loop_info()
        assert mode > 0 and graphs == 1
        for s in slots[:-1]:
            B.release(s)
            assert B.tcd_step(4) > 0
        launched = B.loop_info()[1]
        assert launched == count
        B.release(slots[-1])
        assert B.tcd_step(4) == 0 and B.loop_info()[1:] == (launched, host)
    finally:
        ctx.close()
