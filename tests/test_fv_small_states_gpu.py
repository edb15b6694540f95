"""Batches of many small 1D and 3D finite-volume states: every state as by itself, on both sides of the line between the
generic kernel and the tiles, and no slower than larger states of as many cells."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stepper(gdt, n, nbatch, method="ssp2", flux="burgers"):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), list(n), periodic=True)
    space = gdt.FiniteVolumeSpace(g)
    f = gdt.BurgersFlux() if flux == "burgers" else gdt.LinearTransportFlux([1.0, 0.5, -0.25][:len(n)])
    op = gdt.AdvectionFvOperator(g, gdt.NumericalLaxFriedrichsFlux(f), space)
    u = torch.rand(nbatch * space.num_DoFs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    return gdt.ExplicitRungeKuttaTimeStepper(op, u, method=method), space.num_DoFs


# the tiles (few states, or rows that fill them) and the generic kernel
@pytest.mark.parametrize("n,nbatch", [((2,), 64), ((2,), 40000), ((10,), 40000), ((20,), 40000), ((257,), 500), ((2, 2, 2), 16),
                                      ((2, 2, 2), 8000), ((4, 4, 4), 300), ((4, 4, 4), 1000), ((2, 64, 2), 300),
                                      ((8, 8, 2), 1000), ((32, 4, 4), 300)])
@pytest.mark.parametrize("method,flux", [("ssp2", "burgers"), ("euler", "transport")])
def test_states_of_a_batch_as_by_themselves(gdt, n, nbatch, method, flux):
    batch, cells = _stepper(gdt, n, nbatch, method, flux)
    picked = sorted({0, 1, nbatch // 2, nbatch - 1})
    single = [batch.u[k * cells:(k + 1) * cells].clone() for k in picked]
    dt = 0.1 / max(n) / len(n)
    batch.step(dt, 3)
    for k, u in zip(picked, single):
        gdt.ExplicitRungeKuttaTimeStepper(batch.op, u, method=method).step(dt, 3)
        # a few roundings of values below one per step and face
        assert float((batch.u[k * cells:(k + 1) * cells] - u).abs().max()) <= 1e-14


# as many cells in smaller states: where the tiles were taken for them all the same, 4.0 and 3.0 times as long
@pytest.mark.parametrize("small,large", [(((2,), 200000), ((8,), 50000)), (((2, 2, 2), 8000), ((4, 4, 4), 1000))])
def test_small_states_take_no_longer(gdt, small, large):
    times = []
    for n, nbatch in (small, large):
        st, _ = _stepper(gdt, n, nbatch)
        st.step(1e-6, 20)
        best = float("inf")
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            st.step(1e-6, 50)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times.append(best)
    assert times[0] <= 2.0 * times[1], times
