"""FP64 batches at tight tolerances: teams of several CTAs take as many iterations as one CTA, which always iterates on the
assembled rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element", ["p1", "q1"])
@pytest.mark.parametrize("n", [128, 256, 400])
def test_tight_tolerance_against_one_cta(gdt, n, element):
    mu = torch.tensor(np.exp(np.random.default_rng(n).standard_normal((1, 4))), device="cuda")
    iterations = {}
    for teams in ("cta", "cluster"):
        batch = gdt.BatchedDiffusion([n], element=element).set_teams(teams)
        batch.solve(mu, tol=1e-12)
        iterations[teams] = batch.last_info["max_iterations"]
    assert iterations["cluster"] <= 1.01 * iterations["cta"] + 2
