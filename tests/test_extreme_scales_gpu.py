"""FP64 solves whose coefficients are near the ends of the range of a double: the products that beta is formed from leave it
there, the solution does not."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve(gdt, n, simplex, scale, precond, tol=1e-9):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    kappa = torch.tensor(scale * np.exp(0.3 * np.random.default_rng(1).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    # (constrained rows keep a diagonal of one: the load is zero there)
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    return op.apply_inverse(rhs, opts={"tol": tol, "precond": precond, "max_iter": 5000}), op.last_solve_info


@pytest.mark.parametrize("n,simplex", [([9, 8], False), ([30, 31], True), ([12, 11, 10], True), ([130, 120], False)])
@pytest.mark.parametrize("exponent,precond", [(980, "jacobi"), (600, "none"), (-600, "jacobi"), (-600, "none")])
def test_cg_with_extreme_coefficients(gdt, n, simplex, exponent, precond):
    x, info = _solve(gdt, n, simplex, 2.0**exponent, precond)
    ref, ref_info = _solve(gdt, n, simplex, 1.0, precond, tol=1e-11)
    assert info["converged"] and info["iterations"] <= 1.1 * ref_info["iterations"] + 2
    # both solved to a relative residual of 1e-9 at condition numbers below 1e4
    x = x * 2.0 ** (exponent // 2) * 2.0 ** (exponent - exponent // 2)
    assert float((x - ref).abs().max()) <= 1e-5 * float(ref.abs().max())


@pytest.mark.parametrize("element", ["p1", "q1"])
@pytest.mark.parametrize("exponent", [-980, -500, 500, 900, 980])
def test_batch_with_extreme_coefficients(gdt, element, exponent):
    cells = [8, 33, 16, 64]
    batch = gdt.BatchedDiffusion(cells, element=element)
    kappa = torch.tensor(np.exp(0.3 * np.random.default_rng(2).standard_normal(batch.total_elements)), device="cuda")
    ref = batch.solve(kappa=kappa, tol=1e-9)
    x = batch.solve(kappa=kappa * 2.0**exponent, tol=1e-9)
    # an even power of two: every quantity is scaled exactly
    assert torch.equal(x * 2.0 ** (exponent // 2) * 2.0 ** (exponent - exponent // 2), ref)
