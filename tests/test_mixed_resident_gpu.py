"""Mixed-precision solves of vertex stencils in one launch: rows per thread 1 to 16, matrix entries in shared memory and
beyond it, one-cell-wide grids whose stencil offsets coincide, changed values, the failure paths."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _operator(gdt, n, simplex, mapped):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=simplex)
    if mapped:
        axes = [np.linspace(0.0, 1.0, k + 1) for k in n]
        X = np.stack([a.reshape(-1) for a in np.meshgrid(*axes[::-1], indexing="ij")[::-1]], -1)
        g.map_vertices(X + 0.03 * np.sin(2 * np.pi * X))
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    k = np.exp(np.random.default_rng(4).standard_normal(g.num_elements))
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(torch.tensor(k, device="cuda")))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    return op, rhs


def _solve(op, rhs, form="auto", blocks=0, **opts):
    op.ctx.set_solver_launch(form)
    op.ctx.set_persistent_limits(blocks=blocks)
    try:
        x = op.apply_inverse(rhs, opts={"precision": "mixed", "tol": 1e-11, **opts})
    finally:
        op.ctx.set_solver_launch("auto")
        op.ctx.set_persistent_limits()
    return x, dict(op.last_solve_info)


# slices of 32 rows over 16 warps per block: 36 (Q1 squares) on nine, two and one blocks are 1, 2 and 4 rows per
# thread, 130 (P1 triangles) on two and one 8 and 16; 69 slices of 27 slots on one block exceed its shared
# memory, 378 on three too; [1, 5, 6] has coinciding offsets, 1D three slots
@pytest.mark.parametrize("n,simplex,mapped,blocks", [
    ([37, 29], False, False, 0), ([37, 29], False, False, 2), ([37, 29], False, False, 1), ([64, 63], True, False, 2),
    ([64, 63], True, False, 1), ([11, 10, 9], False, True, 1), ([13, 12, 11], False, True, 1),
    ([24, 22, 20], False, True, 3), ([12, 11, 10], True, False, 0), ([1, 5, 6], True, False, 0), ([31], False, False, 0),
    ([200], False, False, 0), ([2, 2], True, False, 0)])
@pytest.mark.parametrize("precond", ["jacobi", "none"])
def test_resident_matches_graph_and_direct(gdt, n, simplex, mapped, blocks, precond):
    op, rhs = _operator(gdt, n, simplex, mapped)
    xg, ig = _solve(op, rhs, "graph", precond=precond)
    xp, ip = _solve(op, rhs, "auto", blocks, precond=precond)
    assert ip["launch"] == "persistent" and ip["inner_operator"] == "stencil" and ip["converged"]
    # FP32 rounding shifts the sequence by a few per cent between the forms
    assert abs(ig["iterations"] - ip["iterations"]) <= max(3, 0.1 * ig["iterations"])
    rp, col, val = (t.cpu().numpy() for t in op.csr())
    A = sp.csr_matrix((val, col, rp), shape=op.shape)
    b = rhs.cpu().numpy()
    # the stopping test is made on the true residual
    assert np.linalg.norm(b - A @ xp.cpu().numpy()) <= 1.01e-11 * np.linalg.norm(b)
    assert rel_err(xp.cpu().numpy(), spl.spsolve(A.tocsc(), b)) < 1e-8
    xp2, ip2 = _solve(op, rhs, "auto", blocks, precond=precond)
    assert ip2["iterations"] == ip["iterations"] and torch.equal(xp, xp2)


def test_changed_values_and_initial_guess(gdt):
    op, rhs = _operator(gdt, [20, 17], False, False)
    op.csr()[2].mul_(2.0)
    x0 = torch.rand_like(rhs)
    x, info = _solve(op, rhs)
    y = x0.clone()
    op.apply_inverse(rhs, y, opts={"precision": "mixed", "tol": 1e-11})
    assert info["converged"] and op.last_solve_info["converged"]
    assert rel_err(y.cpu().numpy(), x.cpu().numpy()) < 1e-8
    assert float((op.apply(x) - rhs).norm() / rhs.norm()) < 1.01e-11


def test_failures_are_reported(gdt):
    op, rhs = _operator(gdt, [60, 50], True, False)
    with pytest.raises(gdt.GdtError) as e:
        _solve(op, rhs, max_iter=3)
    assert e.value.status == gdt._capi.ENOCONV
    bad = rhs.clone()
    bad[1000] = float("nan")
    with pytest.raises(gdt.GdtError) as e:
        _solve(op, bad)
    assert e.value.status == gdt._capi.ENOCONV
    op.ctx.set_persistent_limits(wait_limit_ns=1)
    try:
        with pytest.raises(gdt.GdtError) as e:
            op.apply_inverse(rhs, opts={"precision": "mixed", "tol": 1e-11})
    finally:
        op.ctx.set_persistent_limits()
    assert e.value.status == gdt._capi.ECUDA and "grid barrier wait ran out" in str(e.value)
    x, info = _solve(op, rhs)
    assert info["converged"] and info["launch"] == "persistent"
