"""Local matrices by quadrature (quad.cuh): every element, form and kind of cell against the
oracle's restatement of the reference's per-point forms.

Sizes leave the kernels' cell groups partly filled: 32 cells per block pass for Q1 and 2D Q2
(1, 31..36 and 64..66 cells), 5 for Q2 hexahedra (1, 8, 27 cells).  The kernels sum over the Gauss
points one direction at a time, the oracle point by point: entries agree to the rounding of some
64 terms, 1e-13 of the largest entry.
"""
import numpy as np
import pytest

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.system import Context, coeffs

pytestmark = pytest.mark.gpu

GALERKIN, SUPG, MASS = 1, 2, 10


@pytest.fixture(scope="module")
def ctx():
    from parmoon_cmg_b200 import _build
    _build.build()
    c = Context(0)
    yield c
    c.close()


def cells_of(sp, n_cells):
    """The first n_cells cells of a space, as a space of its own (all DOFs active)."""
    nbf = (sp["order"] + 1) ** sp["dim"]
    gn = sp["global_numbers"][:n_cells * nbf]
    used, new = np.unique(gn, return_inverse=True)
    nv = 2 ** sp["dim"]
    return dict(dim=sp["dim"], order=sp["order"], coords=sp["coords"][:n_cells * nv * sp["dim"]].copy(),
                global_numbers=new.astype(np.int32).reshape(-1), begin_index=sp["begin_index"][:n_cells + 1],
                n_dof=len(used), n_active=len(used), n_cells=n_cells)


@pytest.mark.parametrize("disc", [GALERKIN, SUPG, MASS])
@pytest.mark.parametrize("warp", [False, True])
@pytest.mark.parametrize("dim,order,n,n_cells", [
    (2, 1, 9, 1), (2, 1, 9, 31), (2, 1, 9, 33), (2, 1, 9, 64),
    (2, 2, 9, 1), (2, 2, 9, 32), (2, 2, 9, 66),
    (3, 1, 4, 1), (3, 1, 4, 36), (3, 1, 4, 64),
    (3, 2, 3, 1), (3, 2, 3, 8), (3, 2, 3, 27),
])
def test_table_coefficients_vs_oracle(ctx, oracle_lib, dim, order, n, n_cells, warp, disc):
    sp = cells_of(mesh.structured_space(dim, order, n), n_cells)
    if warp:
        x = sp["coords"].reshape(-1, dim)
        bend = 0.1 / n * np.sin(5.0 * x[:, ::-1] + 1.0) + 0.3 / n * np.sin(3.0 * x).prod(1, keepdims=True)
        sp["coords"] = np.ascontiguousarray((x + bend).reshape(-1))
    sid = ctx.upload_space(sp)
    nnz = ctx.build_pattern(sid)
    rp, kc = ctx.get_pattern(sid, sp["n_dof"], nnz)
    xq = ctx.quadrature_points(sid, n_cells, dim)
    rng = np.random.default_rng(n_cells + 7 * dim + order)
    tab = rng.uniform(-1.0, 1.0, xq.shape[:-1] + (6,))
    tab[..., 0] = 10.0 ** rng.uniform(-4, 0, xq.shape[:-1])
    ctx.set_coeffs(sid, coeffs(_lib.COEFF_TABLE, delta0=0.7, poly_degree=order), tab)
    ent, rhs = ctx.assemble(sid, disc, sp["n_dof"], nnz)
    co = oracle_lib.coeffs(3, delta0=0.7, order_pd=order)
    ent_o, rhs_o = oracle_lib.assemble(dim, order, disc, sp["coords"], sp["global_numbers"], sp["begin_index"],
                                       sp["n_dof"], sp["n_active"], rp, kc, co, coeff_tab=tab)
    assert np.abs(ent - ent_o).max() <= 1e-13 * np.abs(ent_o).max()
    assert np.abs(rhs - rhs_o).max() <= 1e-13 * np.abs(rhs_o).max()
    # the same again: the sums have a fixed order
    again, rhs2 = ctx.assemble(sid, disc, sp["n_dof"], nnz)
    assert np.array_equal(again, ent) and np.array_equal(rhs2, rhs)
