"""The teams of the batched launch sized by the work: problems on one block and on many, rows beyond a block's shared
memory, more problems than teams, coefficients without a positive diagonal, the bounded waits."""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _solve(gdt, cells, element, kappa, teams=None, blocks=0, **kw):
    ctx = gdt.default_context()
    ctx.set_persistent_limits(blocks=blocks)
    try:
        b = gdt.BatchedDiffusion(cells, element=element)
    finally:
        ctx.set_persistent_limits()
    if teams:
        b.set_teams(teams)
    x, st = b.solve(kappa=kappa, tol=1e-12, keep_stencil=True, **kw)
    return b, x, st


# (sides, blocks): teams of many blocks, of one block, fewer blocks than problems; 200 squares on one block are
# 40,401 rows of which the block's shared memory holds the first 26,624 of one array; 7 rows and less per block
@pytest.mark.parametrize("cells,blocks", [([31], 0), ([1, 2, 3, 5], 0), ([40, 33, 7] * 20, 0), ([17] * 9, 4), ([200], 1),
                                          ([200, 64, 5], 2), ([90, 12], 13)])
@pytest.mark.parametrize("element", ["p1", "q1"])
def test_team_sizes_match_cta_teams(gdt, cells, blocks, element):
    per_cell = 2 if element == "p1" else 1
    k = np.exp(np.random.default_rng(5).standard_normal(sum(per_cell * c * c for c in cells)))
    kappa = torch.tensor(k, device="cuda")
    b, x, st = _solve(gdt, cells, element, kappa, blocks=blocks)
    c, xc, stc = _solve(gdt, cells, element, kappa, teams="cta")
    assert torch.equal(st, stc)  # the same assembly
    ib, rb = b.iterations()
    ic, rc = c.iterations()
    # rounding moves the iteration at which the residual passes 1e-12 by a few per cent
    assert (np.abs(ib - ic) <= np.maximum(2, 0.06 * ic)).all()
    # the true residual ends at 1e-12 or, for the larger sides, where rounding leaves it: no further off than the
    # unscaled iteration of the CTA teams
    assert (rb <= np.maximum(1e-12, 1.5 * rc)).all() and (b.status() == gdt._capi.OK).all()
    for i in range(len(cells)):
        assert rel_err(b.unpack(x, i).cpu().numpy(), c.unpack(xc, i).cpu().numpy()) < 1e-9 if cells[i] > 1 else True
    b2, x2, _ = _solve(gdt, cells, element, kappa, blocks=blocks)
    assert torch.equal(x, x2)  # sums in a fixed order


def test_iteration_limit_and_zero_load(gdt):
    cells = [24, 10, 24]
    kappa = torch.ones(sum(2 * c * c for c in cells), dtype=torch.float64, device="cuda")
    b = gdt.BatchedDiffusion(cells)
    with pytest.raises(gdt.GdtError) as e:
        b.solve(kappa=kappa, tol=1e-12, max_iter=5)
    assert e.value.status == gdt._capi.ENOCONV and (b.iterations()[0] == -6).all()
    x = b.solve(kappa=kappa, force=0.0)
    assert bool((x == 0).all()) and (b.iterations()[0] == 0).all() and b.last_info["all_converged"]


def test_coefficients_that_are_not_positive(gdt):
    # a problem whose diagonal is not positive everywhere stops at the same breakdown as on CTA teams
    cells = [12, 12, 16]
    n = 2 * 144
    k = np.ones(2 * n + 2 * 256)
    k[:n] = -1.0
    for teams in (None, "cta"):
        b = gdt.BatchedDiffusion(cells)
        if teams:
            b.set_teams(teams)
        x = torch.full((b.total_dofs,), 7.0, dtype=torch.float64, device="cuda")
        with pytest.raises(gdt.GdtError) as e:
            b.solve(kappa=torch.tensor(k, device="cuda"), tol=1e-10, x=x)
        assert e.value.status == gdt._capi.ENOCONV
        assert list(b.status()) == [gdt._capi.ENOCONV, gdt._capi.OK, gdt._capi.OK]
        assert b.iterations()[0][0] == -1 and bool((b.unpack(x, 0) == 0).all())


def test_wait_limit_reports_and_recovers(gdt):
    b = gdt.BatchedDiffusion([200])
    mu = torch.ones(4, dtype=torch.float64, device="cuda")
    b.ctx.set_persistent_limits(wait_limit_ns=1)
    try:
        with pytest.raises(gdt.GdtError) as e:
            b.solve(mu)
    finally:
        b.ctx.set_persistent_limits()
    assert e.value.status == gdt._capi.ECUDA and "grid barrier wait ran out" in str(e.value)
    assert list(b.status()) == [gdt._capi.ETIMEOUT]
    b.solve(mu)
    assert b.last_info["all_converged"]
