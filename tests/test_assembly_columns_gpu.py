"""Assembly of 3D Q1 rows by vertex columns against extended-precision element sums, the symmetry of its matrix, and products
of changed values: the CSR schedule and the SELL-32 copy that take turns after a change give the same bits."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu

# edges of the 32-column warps, the 128-column blocks and the z chunks (more than one plane each from 160,000 rows)
SIZES = [(1, 1, 1), (2, 1, 3), (30, 1, 2), (31, 3, 2), (7, 33, 4), (32, 5, 9), (63, 61, 50), (58, 64, 97)]


def _element_sums(n, hi, kappa):
    """{offset (x, y, z): sums over the elements of kappa K on the vertex lattice [z, y, x]} in extended precision."""
    h = [np.longdouble(hi[a]) / n[a] for a in range(3)]
    D = {}
    kap = kappa.reshape(n[::-1]).astype(np.longdouble)
    for i in range(8):
        for j in range(8):
            same = [(i >> a & 1) == (j >> a & 1) for a in range(3)]
            K = np.longdouble(0)
            for a in range(3):
                term = (1 if same[a] else -1) / h[a]
                for c in range(3):
                    if c != a:
                        term = term * h[c] / (3 if same[c] else 6)
                K += term
            off = tuple((j >> a & 1) - (i >> a & 1) for a in range(3))
            arr = D.setdefault(off, np.zeros([k + 1 for k in n[::-1]], np.longdouble))
            x, y, z = i & 1, i >> 1 & 1, i >> 2 & 1
            arr[z:z + n[2], y:y + n[1], x:x + n[0]] += kap * K
    return D


@pytest.mark.parametrize("dirichlet", [True, False])
@pytest.mark.parametrize("n", SIZES)
def test_columns_match_element_sums(gdt, oracle, n, dirichlet):
    rng = np.random.default_rng(sum(n))
    kappa, force = np.exp(rng.standard_normal(np.prod(n))), rng.standard_normal(np.prod(n))
    hi = [1.0, 0.7, 1.9]
    g = gdt.make_cube_grid([0, 0, 0], hi, list(n))
    space = gdt.ContinuousLagrangeSpace(g, 1)
    op = gdt.MatrixOperator(g, space)
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(torch.tensor(kappa, device="cuda")))
    rhs = torch.full((space.num_DoFs,), np.nan, dtype=torch.float64, device="cuda")
    op.assemble(rhs=rhs, force=torch.tensor(force, device="cuda"), dirichlet=dirichlet)
    A, b = oracle.assemble_cg(oracle.grid(3, list(n), 0.0, hi), 1, kappa=kappa, force=force, dirichlet=dirichlet)
    rp, col, val = (t.cpu().numpy().copy() for t in op.csr())
    assert np.array_equal(rp, A.row_ptr) and np.array_equal(col, A.col)
    row = np.repeat(np.arange(A.n), np.diff(rp))
    vn = [k + 1 for k in n]

    def split(v):
        return v % vn[0], v // vn[0] % vn[1], v // (vn[0] * vn[1])

    r, c = split(row), split(col.astype(np.int64))
    bnd_r, bnd_c = (np.any([(q[a] == 0) | (q[a] == n[a]) for a in range(3)], axis=0) for q in (r, c))
    ref = np.empty(len(val), np.longdouble)
    for off, arr in _element_sums(n, hi, kappa).items():
        m = np.all([c[a] - r[a] == off[a] for a in range(3)], axis=0)
        ref[m] = arr[r[2][m], r[1][m], r[0][m]]
    scale = np.abs(ref).max()
    if dirichlet:
        ref[bnd_r | bnd_c] = 0
        ref[bnd_r & (row == col)] = 1
    # an entry: f (9 roundings of terms below 3 f of the diagonal) times a sum of at most 8 coefficients (3 more)
    assert np.abs(val - ref).max() <= 32 * np.finfo(float).eps * scale
    # a load: 8 products with B of sources of either sign
    assert np.abs(rhs.cpu().numpy() - b).max() <= 32 * np.finfo(float).eps * np.abs(force).max() * np.prod(hi) / np.prod(n)
    M = sp.csr_matrix((val, col, rp))
    assert (M != M.T).nnz == 0


@pytest.mark.parametrize("n,simplex", [((9, 8, 7), False), ((40, 38, 41), False), ((21, 20, 23), True), ((60, 59), False)])
def test_changed_values_same_bits(gdt, n, simplex):
    g = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), list(n), simplex=simplex)
    space = gdt.ContinuousLagrangeSpace(g, 1)
    rng = np.random.default_rng(5)
    x = torch.tensor(rng.standard_normal(space.num_DoFs), device="cuda")
    ops = []
    for schedule in (None, 7, 8):
        op = gdt.MatrixOperator(g, space)
        op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(1.0))
        op.assemble(dirichlet=True)
        if schedule is not None:
            op.set_spmv_schedule(schedule)
        op.apply(x)
        ops.append(op)
    factors = rng.uniform(0.5, 2.0, (3, ops[0].nnz))
    for factor in factors:
        for op in ops:
            op.csr()[2].mul_(torch.tensor(factor, device="cuda"))
            op.values_changed()
        rp, col, val = (t.cpu().numpy() for t in ops[0].csr())
        A = sp.csr_matrix((val, col, rp))
        ref, size = A @ x.cpu().numpy(), abs(A) @ abs(x.cpu().numpy())
        staged, copied = ops[1].apply(x), ops[2].apply(x)
        assert torch.equal(staged, copied)
        # the tuned operator goes from one to the other once its products have paid the copy (far below 1001 here)
        first = ops[0].apply(x).clone()
        for _ in range(1001):
            y = ops[0].apply(x)
        # rows of at most 27 products: 27 roundings of sums of at most `size`, on both sides
        for z in (staged, first, y):
            assert (np.abs(z.cpu().numpy() - ref) <= 54 * np.finfo(float).eps * size).all()
        if torch.equal(first, staged):
            assert torch.equal(y, staged)
