"""Launches that the CUDA runtime refuses (a device of which fewer SMs are available): the library runs its other form and
the results stay. The refusal is a fake of the runtime call, preloaded into a process of its own."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKES = {
    # cudaErrorCooperativeLaunchTooLarge
    "cooperative": """
int cudaLaunchCooperativeKernel(const void* f, ...) { (void)f; return 720; }
""",
    # no cluster of the size asked for fits
    "cluster": """
int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* cfg) { (void)f; (void)cfg; *n = 0; return 0; }
""",
}

CHILD = """
import importlib, sys
import numpy as np, torch
gdt = importlib.import_module("dune-gdt_gb300")
out = {}
BODY
np.savez(sys.argv[1], **out)
"""

BATCH = """
cells = [64, 40, 16, 8]
mu = 0.5 + torch.rand(len(cells), 4, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
for element in ("p1", "q1"):
    b = gdt.BatchedDiffusion(cells, element=element)
    for name, teams in (("cluster", "cluster"), ("mixed kinds", ["cluster", "cta", "warp", "cluster"])):
        b.set_teams(teams)
        for k in range(2):
            out[f"{element} {name} {k}"] = b.solve(mu, tol=1e-11).cpu().numpy()
        out[f"{element} {name} status"] = b.status()
    b.set_teams("cluster")
    b.tune(mu)
    out[f"{element} tuned"] = b.solve(mu, tol=1e-11).cpu().numpy()
"""


CG = """
for form in ("auto", "persistent"):
    for n, simplex in (([12], False), ([64, 64], False), ([62, 80], True)):
        g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=simplex)
        prob = gdt.DiffusionProblem(g)
        prob.assemble(torch.ones(g.num_elements, dtype=torch.float64, device="cuda"))
        prob.op.ctx.set_solver_launch(form)
        out[f"{form} {n}"] = prob.op.apply_inverse(prob.rhs, opts={"tol": 1e-11}).cpu().numpy()
        out[f"{form} {n} launch"] = np.array(prob.op.last_solve_info["launch"])
"""


def _run(tmp_path, body, fake=None):
    env = dict(os.environ, PYTHONPATH=ROOT)
    if fake:
        src, lib = tmp_path / f"{fake}.c", tmp_path / f"{fake}.so"
        src.write_text(FAKES[fake])
        subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
        env["LD_PRELOAD"] = str(lib)
    out = tmp_path / f"{fake}.npz"
    r = subprocess.run([sys.executable, "-c", CHILD.replace('BODY', body), str(out)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return dict(np.load(out))


def test_batch_without_cooperative_launch(tmp_path):
    free = _run(tmp_path, BATCH)
    refused = _run(tmp_path, BATCH, "cooperative")
    assert free.keys() == refused.keys()
    for key, x in refused.items():
        if key.endswith("status"):
            assert (x == 0).all()
        else:  # both solved to 1e-11; the condition numbers are below 1e4
            assert np.abs(x - free[key]).max() <= 1e-7 * np.abs(free[key]).max(), key


def test_small_solves_without_cluster_run_on_the_grid(tmp_path):
    free = _run(tmp_path, CG)
    refused = _run(tmp_path, CG, "cluster")
    assert free.keys() == refused.keys()
    for key, x in refused.items():
        if key.endswith("launch"):
            assert str(x) == "persistent", key
        else:
            assert np.abs(x - free[key]).max() <= 1e-7 * np.abs(free[key]).max(), key
