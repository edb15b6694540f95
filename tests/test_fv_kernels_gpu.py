"""The finite-volume kernels at the edges of their tiles, segments and chunks, against the oracle; states of both signs
with zeros; infinities and NaN; more 1D states than a grid dimension holds."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FLUXES = ["burgers", "transport"]
NUMFLUXES = ["lf", "upwind", "eo"]
VELOCITY = (0.7, -0.4, 0.3)


def _operator(gdt, n, flux, num, periodic, boundary):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0 + 0.5 * k for k in range(len(n))], n, periodic=periodic)
    f = gdt.BurgersFlux() if flux == "burgers" else gdt.LinearTransportFlux(VELOCITY[:len(n)])
    nf = {"lf": gdt.NumericalLaxFriedrichsFlux, "upwind": gdt.NumericalUpwindFlux,
          "eo": gdt.NumericalEngquistOsherFlux}[num](f)
    op = gdt.AdvectionFvOperator(g, nf, gdt.FiniteVolumeSpace(g))
    kinds, values = [0] * 6, [0.0] * 6
    if boundary:  # every kind of treatment in turn, sides of one direction treated alike or not
        for side in range(2 * len(n)):
            kinds[side], values[side] = (1, 2, 3)[side % 3], (0.0, 0.3, -0.2)[side % 3]
            t = (gdt.BoundaryTreatmentByCustomExtrapolation(), gdt.BoundaryTreatmentByCustomExtrapolation(0.3),
                 gdt.BoundaryTreatmentByCustomNumericalFlux(-0.2))[side % 3]
            op.append(t, filter=("-x", "+x", "-y", "+y", "-z", "+z")[side])
    return op, kinds, values


def _state(n, seed):
    u = np.random.default_rng(seed).standard_normal(int(np.prod(n)))
    u[::7] = 0.0
    return u


@pytest.mark.parametrize("n", [[2], [255], [256], [257], [1030], [2, 2], [31, 33], [32, 32], [33, 31], [64, 65], [97, 8],
                               [2, 2, 2], [32, 8, 4], [33, 9, 5], [31, 7, 3], [65, 17, 40], [3, 2, 70]])
@pytest.mark.parametrize("periodic,boundary", [(True, False), (False, True), (False, False)])
def test_tile_edges_match_oracle(gdt, oracle, n, periodic, boundary):
    og = oracle.grid(len(n), n, 0.0, [1.0 + 0.5 * k for k in range(len(n))], periodic=periodic)
    u = _state(n, 1)
    ut = torch.tensor(u, device="cuda")
    for fi, flux in enumerate(FLUXES):
        for ni, num in enumerate(NUMFLUXES):
            op, kinds, values = _operator(gdt, n, flux, num, periodic, boundary)
            kw = {"velocity": VELOCITY[:len(n)], "boundary": kinds if boundary else None, "boundary_value": values}
            ref = oracle.fv_apply(og, fi, ni, u, **kw)
            # a handful of roundings of fluxes of size |u|^2 n
            tol = 16 * np.finfo(float).eps * np.abs(u).max() ** 2 * sum(n)
            assert np.abs(op.apply(ut).cpu().numpy() - ref).max() <= tol, (flux, num)
            for method, step in (("ssp2", oracle.fv_ssprk2), ("euler", oracle.fv_explicit_euler)):
                both = torch.cat([ut, 0.5 * ut])  # a batch of two states
                dt = 0.05 / sum(n)
                gdt.ExplicitRungeKuttaTimeStepper(op, both, method=method).step(dt, 3)
                for b, s in enumerate((u, 0.5 * u)):
                    ref = step(og, fi, ni, s, dt, 3, **kw)
                    got = both[b * len(u):(b + 1) * len(u)].cpu().numpy()
                    assert np.abs(got - ref).max() <= 3 * 2 * dt * tol + 16 * np.finfo(float).eps * 4, (flux, num, method)


@pytest.mark.parametrize("n", [[300], [40, 35], [34, 9, 6]])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_nonfinite_states_stay_where_they_spread(gdt, oracle, n, value):
    og = oracle.grid(len(n), n, 0.0, [1.0 + 0.5 * k for k in range(len(n))], periodic=True)
    u = _state(n, 2)
    u[int(np.prod(n)) // 2] = value
    op, _, _ = _operator(gdt, n, "burgers", "lf", True, False)
    got = op.apply(torch.tensor(u, device="cuda")).cpu().numpy()
    ref = oracle.fv_apply(og, 0, 0, u)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    fin = np.isfinite(ref)
    assert np.abs(got[fin] - ref[fin]).max() <= 16 * np.finfo(float).eps * 16 * sum(n)


def test_more_1d_states_than_a_grid_dimension(gdt):
    op, _, _ = _operator(gdt, [4], "burgers", "lf", True, False)
    one = torch.tensor(_state([4], 3), device="cuda")
    many = one.repeat(70000)
    gdt.ExplicitRungeKuttaTimeStepper(op, many, method="ssp2").step(0.01, 2)
    gdt.ExplicitRungeKuttaTimeStepper(op, one, method="ssp2").step(0.01, 2)
    assert torch.equal(many.view(-1, 4), one.expand(70000, 4))
