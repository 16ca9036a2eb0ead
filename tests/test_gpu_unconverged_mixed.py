"""Mixed solves that end at the iteration limit keep their results.

Where damped Jacobi magnifies the upper modes (the mass matrix of trilinear hexahedra, a Galerkin
level whose convection dominates on its cells) a solve stops unconverged, and in the mixed form its
result is what the rounding of the FP32 cycles left: another order of a sum, or the coarse levels in
another precision, moves it by 1e-7 to 1e-4.  The golden entries are those of the library that
launches every coarse level in FP32 and adds Gram-Schmidt sums over blocks of 256 rows; the bound is
the 1e-9 within which an unchanged call's result is to stay.  ``python tests/test_gpu_unconverged_mixed.py
FILE`` writes the entries of the library at hand.
"""
import json
import os

import numpy as np
import pytest

from parmoon_cmg_b200 import mesh
from parmoon_cmg_b200.system import GALERKIN, SUPG, TSystemCD3D, TSystemTCD3D, coeffs, solver_params

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_unconverged.json")
PRM = dict(precision=1, stop_rule=1, red_factor=1e-10, maxit=300)


def _step(n0, levels, eps):
    spaces, parents = mesh.structured_hierarchy(3, 1, n0, levels)
    S = TSystemTCD3D(spaces, parents)
    S.Init(coeffs(0, eps=eps, b=(0.5, 0.3, -0.4), f=0.25))
    u = np.exp(-((mesh.dof_coords(spaces[-1]) - 0.35) ** 2).sum(1) / (2 * 0.08 ** 2))
    S.AssembleMRhs(u)
    S.AssembleARhs()
    info = S.Step(u, 1e-3, 0.5, 0.5, 0.5, 0.5, params=solver_params(**PRM))
    return u, info


def _galerkin(n0, levels, eps):
    spaces, parents = mesh.structured_hierarchy(3, 2, n0, levels)
    S = TSystemCD3D(spaces, parents, disctype=GALERKIN, coarse_disctype=SUPG)
    S.Init(coeffs(0, eps=eps, b=(0.6, 0.64, 0.48), f=1.0, delta0=1.0 / 3.0))
    u, rhs = np.zeros(S.N_DOF), np.zeros(S.N_DOF)
    S.Assemble(u, rhs)
    info = S.Solve(u, rhs, solver_params(**PRM))
    return u, info


CASES = {
    "step_q1_32": lambda: _step(2, 5, 1e-3),
    "step_q1_48": lambda: _step(3, 5, 1e-2),
    "galerkin_q2_8": lambda: _galerkin(2, 3, 1e-2),
    "galerkin_q2_12": lambda: _galerkin(3, 3, 1e-2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_unconverged_mixed_result(name):
    with open(GOLDEN) as f:
        want = json.load(f)[name]
    u, info = CASES[name]()
    assert info.status != 0 and info.iterations == 300
    entries = np.array(want["entries"])
    assert np.linalg.norm(u[::want["stride"]] - entries) <= 1e-9 * np.linalg.norm(entries)
    assert abs(np.linalg.norm(u) - want["norm"]) <= 1e-9 * want["norm"]


if __name__ == "__main__":
    import sys
    out = {}
    for name, run in CASES.items():
        u, info = run()
        stride = max(1, u.size // 200)
        out[name] = dict(stride=stride, norm=float(np.linalg.norm(u)), entries=[float(v) for v in u[::stride]])
        print(name, info.iterations, info.status, info.final_residual / info.initial_residual)
    with open(sys.argv[1], "w") as f:
        json.dump(out, f)
