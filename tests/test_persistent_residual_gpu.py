"""FP64 CG of small systems on one cluster and on the grid: true residual and solution, checked on the host against the
assembled matrix and a direct solve."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


# 1 slice to 160 (the largest on a cluster), one and two slices per warp, and one system beyond that
@pytest.mark.parametrize("precond", ["jacobi", "none"])
@pytest.mark.parametrize("form", ["cluster", "grid"])
@pytest.mark.parametrize("n,simplex", [((3,), False), ((200,), False), ((6, 5), True), ((40, 33), False), ((70, 70), True),
                                       ((9, 8, 11), False), ((15, 18, 15), True), ((63, 79), False), ((62, 80), True),
                                       ((63, 80), False)])
def test_true_residual_and_solution(gdt, n, simplex, form, precond):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), list(n), simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    kappa = torch.tensor(np.exp(np.random.default_rng(8).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    op.ctx.set_persistent_limits(wait_limit_ns=2_000_000_000 if form == "grid" else 0)  # a limit of the caller's is the grid's
    try:
        x = op.apply_inverse(rhs, opts={"tol": 1e-11, "precond": precond, "max_iter": 30000}).cpu().numpy()
    finally:
        op.ctx.set_persistent_limits()
    assert op.last_solve_info["launch"] == "persistent" and op.last_solve_info["converged"]
    rp, col, val = (t.cpu().numpy() for t in op.csr())
    A, b = sp.csr_matrix((val, col, rp), shape=op.shape), rhs.cpu().numpy()
    lu = spl.splu(A.tocsc())
    exact = lu.solve(b)
    exact += lu.solve(b - A @ exact)
    # the recurrence stops at 1e-11 |b|; the true residual leaves it by the rounding of the iterates, a small multiple
    # of eps |A| |x| (Greenbaum 1997)
    floor = 16 * 2.0**-53 * spl.norm(A, np.inf) * np.linalg.norm(exact)
    assert np.linalg.norm(b - A @ x) <= 1.01e-11 * np.linalg.norm(b) + floor
    # and the solution by the inverse's norm times that, for systems of a condition number below 1e5 (2D and 3D)
    if len(n) > 1:
        assert rel_err(x, exact) <= 1e-6
