"""The forms of the persistent FP64 CG launch: slices per warp 1 to 16 in registers, vectors in memory beyond
that, matrix entries partly in shared memory, exact zeros left out, blocks and warps without rows."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _system(gdt, dim, n, simplex, dg, unit):
    g = gdt.make_cube_grid([0.0] * dim, [1.0] * dim, n, simplex=simplex)
    k = np.random.default_rng(3).standard_normal(g.num_elements)
    prob = gdt.DiffusionProblem(g, dg=dg)
    prob.assemble(torch.tensor(np.ones_like(k) if unit else np.exp(k), device="cuda"))
    return prob.op, prob.rhs


def _solve(op, rhs, form, blocks=0, **opts):
    op.ctx.set_solver_launch(form)
    op.ctx.set_persistent_limits(blocks=blocks)
    try:
        x = op.apply_inverse(rhs, opts={"tol": 1e-12, "max_iter": 100000, **opts})
    finally:
        op.ctx.set_solver_launch("auto")
        op.ctx.set_persistent_limits()
    return x, dict(op.last_solve_info)


# (grid, blocks): 36 slices of Q1 squares on 5, 3, 2 and 1 blocks are 1, 2, 4 and 8 slices per warp; the 130
# slices of P1 triangles on one block are 17 (vectors in memory), on two 9 (16); 42 slices of 27-entry rows on one
# block exceed its shared memory; single-slice, single-element and 1D systems leave warps without rows
@pytest.mark.parametrize("dim,n,simplex,dg,blocks", [
    (2, [37, 29], False, False, 5), (2, [37, 29], False, False, 3), (2, [37, 29], False, False, 2),
    (2, [37, 29], False, False, 1), (2, [64, 63], True, False, 1), (2, [64, 63], True, False, 2),
    (3, [11, 10, 9], False, False, 1), (3, [11, 10, 9], False, False, 0), (3, [7, 6, 5], True, False, 0),
    (2, [9, 7], True, True, 1), (2, [2, 2], False, False, 0), (1, [31], False, False, 0), (1, [32], False, False, 0)])
@pytest.mark.parametrize("precond,unit", [("jacobi", False), ("none", True)])
def test_persistent_forms_match_graph_and_direct(gdt, dim, n, simplex, dg, blocks, precond, unit):
    op, rhs = _system(gdt, dim, n, simplex, dg, unit)
    xg, ig = _solve(op, rhs, "graph", precond=precond)
    xp, ip = _solve(op, rhs, "persistent", blocks, precond=precond)
    assert ip["launch"] == "persistent" and ig["launch"] == "graph" and ip["converged"]
    assert abs(ig["iterations"] - ip["iterations"]) <= max(2, 0.02 * ig["iterations"])
    rp, col, val = (t.cpu().numpy() for t in op.csr())
    xd = spl.spsolve(sp.csr_matrix((val, col, rp), shape=op.shape).tocsc(), rhs.cpu().numpy())
    # both stop at a relative residual of 1e-12; the condition numbers here are below 1e4
    assert rel_err(xp.cpu().numpy(), xd) < 1e-8 and rel_err(xg.cpu().numpy(), xd) < 1e-8
    xp2, ip2 = _solve(op, rhs, "persistent", blocks, precond=precond)
    assert ip2["iterations"] == ip["iterations"] and torch.equal(xp, xp2)


def test_product_after_persistent_solve_keeps_zero_entries(gdt):
    # the solve leaves exact zeros out of its copy of the matrix; a product afterwards still multiplies them
    # (0 * inf is NaN in the rows coupled to that column)
    op, rhs = _system(gdt, 2, [12, 11], True, False, True)
    op.set_spmv_schedule(8)
    x = torch.ones_like(rhs)
    x[40] = float("inf")
    before = op.apply(x)
    _solve(op, rhs, "persistent")
    after = op.apply(x)
    assert torch.equal(torch.isnan(before), torch.isnan(after)) and bool(torch.isnan(after).any())
    fin = torch.isfinite(before)
    assert torch.equal(before[fin], after[fin])


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_persistent_reports_nonfinite_right_hand_side(gdt, value):
    op, rhs = _system(gdt, 2, [20, 20], False, False, False)
    bad = rhs.clone()
    bad[100] = value
    for form in ("graph", "persistent"):
        with pytest.raises(gdt.GdtError) as e:
            _solve(op, bad, form)
        assert e.value.status == gdt._capi.ENOCONV
