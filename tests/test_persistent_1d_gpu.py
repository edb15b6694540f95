"""FP64 CG on 1D grids with a constant coefficient: the persistent launch ends after n / 2 iterations, when the mirrored
halves of the residual meet, and with the solution of a direct solve."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 160 slices or less on one cluster (4,001), one and two slices per warp on the grid, vectors in memory on few blocks
@pytest.mark.parametrize("n,blocks", [(1000, 0), (4001, 0), (10000, 0), (20000, 0), (10000, 2)])
@pytest.mark.parametrize("precond", ["jacobi", "none"])
def test_constant_coefficient_ends_after_half_the_cells(gdt, n, blocks, precond):
    g = gdt.make_cube_grid([0.0], [1.0], [n])
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(1.0))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    op.ctx.set_persistent_limits(blocks=blocks)
    try:
        x = op.apply_inverse(rhs, opts={"tol": 1e-12, "precond": precond, "max_iter": n // 2 + 10})
    finally:
        op.ctx.set_persistent_limits()
    info = op.last_solve_info
    assert info["launch"] == "persistent" and info["converged"]
    assert abs(info["iterations"] - n // 2) <= 1
    t = torch.arange(n + 1, dtype=torch.float64, device="cuda") / n
    exact = t * (1 - t) / 2  # linear elements are exact in the nodes
    # an iteration count of n / 2 and an error of eps times that per step
    assert float((x - exact).abs().max() / exact.max()) <= 2.2e-16 * n * n / 2
