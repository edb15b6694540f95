"""Finite volumes with a cell that is not a number: one Euler step reaches the neighbours whose faces take that cell's state,
and no others, in every dimension (tiles, and the generic kernel for many small states)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# faces in +x take: the state upwind of them; the upper state where the mean is not positive (NaN); EO none that is not
# positive (NaN)
@pytest.mark.parametrize("flux,num,velocity,reached", [
    ("transport", "Upwind", 1.0, (0, 1)), ("transport", "Upwind", -1.0, (-1, 0)), ("transport", "EngquistOsher", 1.0, (0,)),
    ("burgers", "Upwind", None, (-1, 0)), ("burgers", "EngquistOsher", None, (0,))])
@pytest.mark.parametrize("n,nbatch", [((300,), 1), ((70, 41), 1), ((40, 9, 11), 1), ((6,), 60000), ((6, 4, 4), 3000)])
def test_nan_reaches_the_faces_that_take_it(gdt, n, nbatch, flux, num, velocity, reached):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), list(n), periodic=True)
    space = gdt.FiniteVolumeSpace(g)
    f = gdt.BurgersFlux() if flux == "burgers" else gdt.LinearTransportFlux([velocity] * len(n))
    op = gdt.AdvectionFvOperator(g, getattr(gdt, f"Numerical{num}Flux")(f), space)
    shape = (nbatch, *n[::-1])
    u = 0.5 + torch.rand(shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    cell = (nbatch // 2, *(k // 2 for k in n[::-1]))
    u[cell] = float("nan")
    expected = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for axis in range(1, len(n) + 1):
        for k in reached:
            at = list(cell)
            at[axis] += k
            expected[tuple(at)] = True
    flat = u.reshape(-1)
    gdt.ExplicitRungeKuttaTimeStepper(op, flat, method="euler").step(1e-4)
    assert torch.equal(torch.isnan(flat).reshape(shape), expected)
