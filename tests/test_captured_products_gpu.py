"""Products captured in a CUDA graph of the caller: replays stay right whatever solves run in between."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(gdt, n, simplex=True):
    stream = torch.cuda.Stream()
    ctx = gdt.Context(stream=stream)
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space, ctx=ctx)
    kappa = torch.tensor(np.exp(np.random.default_rng(6).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    torch.cuda.synchronize()
    return op, rhs, stream


# the solve keeps its rows in registers (0 and 2 blocks), or streams 16-bit columns (1 block), and leaves zeros out
@pytest.mark.parametrize("precision,blocks", [("fp64", 0), ("fp64", 2), ("fp64", 1), ("mixed", 0)])
def test_replayed_product_after_solves(gdt, precision, blocks):
    op, rhs, stream = _system(gdt, [64, 63])
    op.set_spmv_schedule(8)  # the product reads its SELL-32 copy
    x = torch.randn(rhs.numel(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    y = torch.zeros_like(rhs)
    torch.cuda.synchronize()
    expected = op.apply(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        op.apply(x, y)
    op.ctx.set_persistent_limits(blocks=blocks)
    op.apply_inverse(rhs, opts={"precision": precision, "tol": 1e-10})
    assert op.last_solve_info["launch"] == "persistent"
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, expected)
    assert torch.equal(op.apply(x), expected)
