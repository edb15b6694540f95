"""FP64 CG of small systems on one cluster: the same solution and iteration counts as the same launch on the grid (a wait
limit of the caller's chooses that), up to and beyond the largest that takes the cluster."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(gdt, n, simplex, seed=3):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), list(n), simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    kappa = torch.tensor(np.exp(np.random.default_rng(seed).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    return op, rhs


# 1 slice, a block without rows in its last warps, one and two slices per warp, 160 slices (5,120 rows) and more
@pytest.mark.parametrize("precond", ["jacobi", "none"])
@pytest.mark.parametrize("n,simplex", [((3,), False), ((200,), False), ((6, 5), True), ((40, 33), False), ((70, 70), True),
                                       ((9, 8, 11), False), ((15, 15, 15), False), ((15, 18, 15), True),
                                       ((63, 79), False), ((62, 80), True), ((63, 80), False)])
def test_cluster_matches_grid(gdt, n, simplex, precond):
    op, rhs = _problem(gdt, n, simplex)
    opts = {"tol": 1e-11, "precond": precond, "max_iter": 30000}
    x = op.apply_inverse(rhs, opts=opts)
    info = op.last_solve_info
    op.ctx.set_persistent_limits(wait_limit_ns=2_000_000_000)
    try:
        y = op.apply_inverse(rhs, opts=opts)
    finally:
        op.ctx.set_persistent_limits()
    grid = op.last_solve_info
    assert info["launch"] == grid["launch"] == "persistent" and info["converged"] and grid["converged"]
    assert abs(info["iterations"] - grid["iterations"]) <= max(2, 0.02 * grid["iterations"])
    # both residuals are at most 1e-11 |b|, or at the rounding floor of the iteration (1D), the same for both
    floor = max(info["rel_residual"], grid["rel_residual"], 1e-11)
    assert float(op.apply(x - y).norm()) <= 4 * floor * float(rhs.norm())
    z = op.apply_inverse(rhs, opts=opts)
    assert torch.equal(x, z)


def test_contexts_in_threads(gdt):
    """Solves of contexts of their own in several threads, each with its kept memory and stream."""
    results = {}

    def work(k):
        ctx = gdt.Context()
        g = gdt.make_cube_grid([0.0, 0.0], [1.0, 1.0], [40 + 50 * k, 60])
        space = gdt.ContinuousLagrangeSpace(g, 1)
        op = gdt.MatrixOperator(g, space, ctx=ctx)
        op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(1.0))
        rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
        op.assemble(rhs=rhs, force=1.0, dirichlet=True)
        results[k] = [op.apply_inverse(rhs, opts={"tol": 1e-11, "precision": p}) for p in ["fp64"] * 5]
        results[-k - 1] = [op.apply_inverse(rhs, opts={"tol": 1e-11, "precision": p}) for p in ["mixed"] * 5]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(results) == 8
    for xs in results.values():
        for x in xs[1:]:
            assert torch.equal(x, xs[0])
