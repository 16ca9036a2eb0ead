"""A coefficient table is the caller's again when set_coeffs returns, also in page-locked memory and
with work queued on the context's stream."""
import numpy as np
import pytest
import torch

from parmoon_cmg_b200 import _lib, mesh
from parmoon_cmg_b200.system import GALERKIN, Context, coeffs

pytestmark = pytest.mark.gpu


def test_page_locked_table_refilled_after_set_coeffs():
    spaces, _ = mesh.structured_hierarchy(3, 2, 12, 1)
    sp = spaces[0]

    def assembled(table, refill, busy):
        ctx = Context(0)
        try:
            sid = ctx.upload_space(sp)
            nnz = ctx.build_pattern(sid)
            ctx.set_coeffs(sid, coeffs(0, eps=0.1, f=1.0))
            ctx.assemble(sid, GALERKIN, sp["n_dof"], nnz)
            if busy:  # some 25 ms in front of the copy
                with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
                    torch.cuda._sleep(50_000_000)
            ctx.set_coeffs(sid, coeffs(_lib.COEFF_TABLE), table)
            if refill:
                table[:] = 7.0
            return ctx.assemble(sid, GALERKIN, sp["n_dof"], nnz)
        finally:
            ctx.close()

    rng = np.random.default_rng(3)
    values = rng.uniform(0.5, 1.5, (sp["n_cells"], 64, 6))
    want = assembled(values.copy(), False, False)
    pinned = torch.from_numpy(values).pin_memory().numpy()
    got = assembled(pinned, True, True)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
