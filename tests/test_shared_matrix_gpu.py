"""One matrix used from several threads, each with a context and stream of its own: products keep their bits while FP64 and
mixed-precision solves run, and the solves theirs."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,simplex", [([90, 80], True), ([22, 23, 21], False)])
def test_products_and_solves_in_threads(gdt, n, simplex):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    ctx = [gdt.Context(stream=torch.cuda.Stream()) for _ in range(4)]
    op = gdt.MatrixOperator(g, space, ctx=ctx[0])
    kappa = torch.tensor(np.exp(np.random.default_rng(1).standard_normal(g.num_elements)), device="cuda")
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    rhs = torch.zeros(space.num_DoFs, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    op.assemble(rhs=rhs, force=1.0, dirichlet=True)
    op.set_spmv_schedule(8)  # the products read the SELL-32 copy
    x = torch.rand(space.num_DoFs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    torch.cuda.synchronize()
    product = op.apply(x)
    solution = {p: op.apply_inverse(rhs, opts={"tol": 1e-10, "precision": p}) for p in ("fp64", "mixed")}
    torch.cuda.synchronize()
    lib = gdt._capi.load()
    wrong = []

    def multiply(k):
        y = torch.empty_like(rhs)
        torch.cuda.synchronize()
        for i in range(300):
            st = lib.gdt_spmv(ctx[k].handle, op.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()))
            ctx[k].synchronize()
            if st != gdt._capi.OK or not torch.equal(y, product):
                wrong.append(("product", i, st))
                return

    def solve(k, precision):
        opts, info = gdt.MatrixOperator._solver_opts({"tol": 1e-10, "precision": precision}), gdt._capi.SolveInfo()
        for i in range(10):
            y = torch.zeros_like(rhs)
            torch.cuda.synchronize()
            st = lib.gdt_solve(ctx[k].handle, op.handle, C.c_void_p(rhs.data_ptr()), C.c_void_p(y.data_ptr()), C.byref(opts),
                               C.byref(info))
            if st != gdt._capi.OK or not torch.equal(y, solution[precision]):
                wrong.append((precision, i, st))
                return

    threads = [threading.Thread(target=multiply, args=(0,)), threading.Thread(target=solve, args=(1, "fp64")),
               threading.Thread(target=solve, args=(2, "fp64")), threading.Thread(target=solve, args=(3, "mixed"))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
