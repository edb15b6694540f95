"""FP64 CG in one launch on rows of more than 32 entries, and streaming with 16-bit and 32-bit columns: the same solution
and iteration counts as the graph form, on few blocks too (several slices per warp, streaming) and with blocks
without rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve(op, rhs, launch, blocks=0, precond="jacobi"):
    op.ctx.set_solver_launch(launch)
    lib = op.ctx.lib
    if blocks:
        assert lib.gdt_context_set_persistent_limits(op.ctx.handle, blocks, 0) == 0
    try:
        x = op.apply_inverse(rhs, opts={"tol": 1e-11, "precond": precond})
    finally:
        op.ctx.set_solver_launch("auto")
        lib.gdt_context_set_persistent_limits(op.ctx.handle, 0, 0)
    return x, op.last_solve_info


# 27 entries for cells up to 125 for vertices: 1 cell; a block per slice; resident with several slices per warp; streaming on
# few blocks
@pytest.mark.parametrize("n,blocks,precond", [((1, 1, 1), 0, "jacobi"), ((2, 3, 1), 0, "none"), ((5, 4, 7), 0, "jacobi"),
                                              ((12, 13, 11), 0, "jacobi"), ((12, 13, 11), 3, "jacobi"),
                                              ((14, 9, 13), 1, "none"), ((24, 25, 23), 0, "jacobi")])
def test_long_rows_match_graph(gdt, n, blocks, precond):
    g = gdt.make_cube_grid([0.0] * 3, [1.0] * 3, list(n))
    space = gdt.ContinuousLagrangeSpace(g, 2)
    op = gdt.MatrixOperator(g, space)
    kappa = torch.tensor(np.exp(np.random.default_rng(3).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    xg, ig = _solve(op, rhs, "graph", precond=precond)
    xp, ip = _solve(op, rhs, "auto", blocks, precond)
    assert ig["launch"] == "graph" and ip["launch"] == "persistent" and ip["converged"]
    assert abs(ip["iterations"] - ig["iterations"]) <= max(2, 0.02 * ig["iterations"])
    # both residuals are at most 1e-11 |b| (or at their rounding floor, far below): the difference of the residuals
    # is what A (x - y) may be
    r = op.apply(xp - xg)
    assert float(r.norm()) <= 4e-11 * float(rhs.norm())
    xr, _ = _solve(op, rhs, "auto", blocks, precond)
    assert torch.equal(xp, xr)


# more than 128 slices per block: 16-bit differences (bands up to 32,767, here at most 3,162) and 32-bit columns (36,673);
# q in shared memory (up to about 22,000 rows a block) and not
@pytest.mark.parametrize("n,blocks", [((50, 61, 70), 40), ((50, 61, 70), 2), ((190, 190, 2), 20), ((190, 190, 2), 3)])
def test_streaming_columns(gdt, n, blocks):
    g = gdt.make_cube_grid([0.0] * 3, [1.0] * 3, list(n))
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    kappa = torch.tensor(np.exp(np.random.default_rng(3).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    xg, ig = _solve(op, rhs, "graph")
    xp, ip = _solve(op, rhs, "auto", blocks)
    assert ig["launch"] == "graph" and ip["launch"] == "persistent" and ip["converged"]
    assert abs(ip["iterations"] - ig["iterations"]) <= max(2, 0.02 * ig["iterations"])
    r = op.apply(xp - xg)
    assert float(r.norm()) <= 4e-11 * float(rhs.norm())
