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


# The products with changed values read the CSR arrays until the copy would have paid its fill; whichever of them is
# captured, and not replayed, the next one must not take the copy for filled
def test_captured_fill_does_not_count_as_done(gdt):
    op, rhs, stream = _system(gdt, [97, 101, 53], simplex=False)
    x = torch.randn(rhs.numel(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    y = torch.zeros_like(rhs)
    torch.cuda.synchronize()
    op.apply(x)  # tunes
    val = op.csr()[2]
    # the fill falls due at an even or an odd product: with one product more in front a captured one meets it
    for schedule, before in ((None, 0), (None, 1), (8, 0)):
        if schedule is not None:
            op.set_spmv_schedule(schedule)
        with torch.cuda.stream(stream):
            expected = 2.0 * op.apply(x)  # a power of two: the same bits scaled
            val *= 2.0
        op.values_changed()
        stream.synchronize()
        for k in range(before):
            op.apply(x)
        for k in range(60):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                op.apply(x, y)
            got = op.apply(x)
            torch.cuda.synchronize()
            # (the schedules add in different orders)
            assert float((got - expected).abs().max()) <= 1e-12 * float(expected.abs().max()), (schedule, k)
            if k % 8 == 7:
                graph.replay()
                torch.cuda.synchronize()
                assert float((y - expected).abs().max()) <= 1e-12 * float(expected.abs().max()), (schedule, k)


# Tuning anew may choose another schedule; the copy that a captured product reads stays
@pytest.mark.parametrize("n,simplex", [([64, 63], True), ([17], False), ([30, 29, 31], False)])
def test_replayed_product_after_tuning_anew(gdt, n, simplex):
    op, rhs, stream = _system(gdt, n, simplex)
    op.set_spmv_schedule(8)
    x = torch.randn(rhs.numel(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    y = torch.zeros_like(rhs)
    torch.cuda.synchronize()
    expected = op.apply(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        op.apply(x, y)
    for _ in range(3):
        assert gdt._capi.load().gdt_matrix_tune(op.ctx.handle, op.handle, None, None) == gdt._capi.OK
        stream.synchronize()
        y.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, expected)
