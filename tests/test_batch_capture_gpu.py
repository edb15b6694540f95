"""A batch's first solve captured in a CUDA graph of the caller, without waiting: nothing is allocated by a solve."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,teams", [("fp64", "cluster"), ("fp64", "cta"), ("fp64", "warp"), ("mixed", "cluster"),
                                             ("mixed", "cta"), ("fp64", ["cluster", "cta", "warp", "cluster"])])
@pytest.mark.parametrize("element", ["p1", "q1"])
def test_first_solve_captured(gdt, precision, teams, element):
    stream = torch.cuda.Stream()
    cells = [64, 40, 16, 8]
    mu = 0.5 + torch.rand(len(cells), 4, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    batch = [gdt.BatchedDiffusion(cells, ctx=gdt.Context(stream=stream), element=element).set_teams(teams) for _ in range(2)]
    x = [torch.zeros(b.total_dofs, dtype=torch.float64, device="cuda") for b in batch]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        batch[0].solve(mu, x=x[0], precision=precision, wait=False)
    for _ in range(2):
        x[0].zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert (batch[0].status() == gdt._capi.OK).all()
        batch[1].solve(mu, x=x[1], precision=precision)
        assert torch.equal(x[0], x[1])
