"""FP64 CG with rows in registers: blocks that hold more entries than their shared memory takes and have fewer slices than
their warps have slots, the last block of the grid among them (its empty slots lie beyond the slice table)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# On 152 SMs: SWIPDG of 200^2 squares (7,500 slices, at most 50 in a block of 64 slots with 18,000 entries), of 256^2
# (12,288 slices, at most 81 of 128) and 253,638 rows of 27 entries without constraints (7,927 slices, at most 53 of
# 64). The table ends with the last block's slices.
@pytest.mark.parametrize("n,dg,slices", [([200, 200], True, 7500), ([256, 256], True, 12288), ([60, 62, 65], False, 7927)])
def test_full_blocks_with_empty_slots_match_graph(gdt, n, dg, slices):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=dg)
    kappa = torch.tensor(np.exp(np.random.default_rng(5).standard_normal(g.num_elements)), device="cuda")
    if dg:
        prob = gdt.DiffusionProblem(g, dg=True)
        prob.assemble(kappa)
        op, rhs = prob.op, prob.rhs
    else:  # a diffusion matrix with a reaction term in place of boundary conditions: every row keeps its 27 entries
        space = gdt.ContinuousLagrangeSpace(g, 1)
        op = gdt.MatrixOperator(g, space)
        op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
        rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
        op.assemble(rhs=rhs, force=1.0)
        rp, col, val = op.csr()
        row = torch.repeat_interleave(torch.arange(space.num_DoFs, device="cuda"), (rp[1:] - rp[:-1]).long())
        val[col == row] *= 1.5
        op.values_changed()
    assert (op.shape[0] + 31) // 32 == slices
    x = {}
    for form in ("graph", "persistent"):
        op.ctx.set_solver_launch(form)
        try:
            x[form] = op.apply_inverse(rhs, opts={"tol": 1e-8, "max_iter": 50000})
        finally:
            op.ctx.set_solver_launch("auto")
        assert op.last_solve_info["launch"] == form and op.last_solve_info["converged"]
        x[form, "iterations"] = op.last_solve_info["iterations"]
        # the recurrence stops at 1e-8 |b|; rounding separates it from the true residual by eps times the condition number
        # (at most about 1e7 here) and much less than that on average
        assert float((rhs - op.apply(x[form])).norm()) <= 2e-8 * float(rhs.norm())
    assert abs(x["graph", "iterations"] - x["persistent", "iterations"]) <= max(2, 0.02 * x["graph", "iterations"])
