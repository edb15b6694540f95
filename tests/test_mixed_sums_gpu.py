"""The sums of the mixed-precision solves: FP32 products, added in FP64 from a thread's value on in both launch forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_products_of_a_warp_are_added_in_fp64(gdt):
    # A diagonal matrix of 32 x 32 rows with 1 + 2^-23 and 1 in turn, right-hand side 1, no preconditioner: p.q is
    # 1024 (1 + 2^-24) and alpha = 1 - 2^-24 in FP32. Added in FP32 over a warp, 32 + 2^-19 is rounded to 32 and alpha
    # is 1. The first step leaves a residual of 6e-8, so the solve ends with x = alpha.
    g = gdt.make_cube_grid([0.0, 0.0], [1.0, 1.0], [31, 31])
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(1.0))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0)
    rp, col, val = op.csr()
    n = space.num_DoFs
    assert n == 1024
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    val.copy_(torch.where(col == row, 1.0 + 2.0**-23 * (1 - row % 2), 0.0))
    op.values_changed()
    x = {}
    for form in ("graph", "auto"):
        op.ctx.set_solver_launch(form)
        try:
            x[form] = op.apply_inverse(torch.ones_like(rhs), opts={"precision": "mixed", "precond": "none", "tol": 1e-6})
        finally:
            op.ctx.set_solver_launch("auto")
        assert op.last_solve_info["iterations"] == 1 and op.last_solve_info["inner_operator"] == "stencil"
        assert op.last_solve_info["launch"] == ("graph" if form == "graph" else "persistent")
        assert torch.equal(x[form], torch.full_like(rhs, 1.0 - 2.0**-24))
