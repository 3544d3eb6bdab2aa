"""The row walks as they run on large meshes -- vector P2 by default, where a warp
takes several groups of nodes one after the other, and one warp a vertex group
(more than 1,480 groups) for P1, P2 and P3 -- against the scatter; and all of
them against the oracle on small ones.

Element matrices are positive semi-definite: an entry's |contributions| sum to
at most sqrt(A_ii A_jj), of which the two orders of summation differ by less
than 1e-12 (some tens of terms at 2^-53; FP32 vector P2 adds the same rounded
entries), and an element's own rounding is below 1e-14 of the largest entry."""
import numpy as np
import pytest

from conftest import ensure_library
from gpu_util import run_system, tolerance_check
from oracle import fem_oracle as fo

pytestmark = pytest.mark.gpu

SPACE = {"p1": ("P", 1), "p2": ("P", 2), "p3": ("P", 3), "vp2": ("P", 2, (3,))}


@pytest.mark.parametrize("kind,coef,n,order", [("p1", "p1", 36, "permuted"), ("p1", "dg0", 47, "natural"), ("p2", "p1", 36, "natural"),
                                               ("p2", "dg0", 37, "permuted"), ("p3", "dg0", 36, "natural"),
                                               ("vp2", "dg0", 33, "natural"), ("vp2", "dg0", 33, "permuted")])
def test_large_meshes_match_the_scatter(kind, coef, n, order):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    rng = np.random.default_rng(n)
    cells = m.cells if order == "natural" else rng.permuted(m.cells[rng.permutation(m.num_cells)], axis=1)
    mesh = fem.Mesh(m.geometry_x, cells, grid_n=n)
    V = fem.functionspace(mesh, SPACE[kind])
    Q = fem.functionspace(mesh, ("DG", 0) if coef == "dg0" else ("P", 1))
    k, mu = (fem.Function(Q, np.exp(rng.standard_normal(Q.num_nodes))) for _ in range(2))
    a = cx.form(fem.elasticity(V, k, mu, precision="fp32") if kind == "vp2" else fem.stiffness(V, k))
    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    rp, col, _ = A.device_csr()
    N = len(rp) - 1
    row = torch.repeat_interleave(torch.arange(N, device="cuda"), (rp[1:] - rp[:-1]).long())
    col = col.long()
    other = "coalesced" if kind == "vp2" else "atomic-full"
    asm.assemble_matrix(a, R, variant=other)
    d = torch.zeros(N, dtype=torch.float64, device="cuda")
    d[row[row == col]] = R.values[row == col]
    tol = 1e-12 * torch.sqrt(d[row] * d[col]) + 1e-14 * R.values.abs().max()
    dofs = fem.locate_boundary_dofs(V)[::2]
    mark = torch.zeros(N, dtype=torch.bool, device="cuda")
    mark[torch.as_tensor(np.asarray(dofs), device="cuda").long()] = True
    for bcs in ([], [fem.dirichletbc(0.0, dofs, V)]):
        A.values.fill_(float("nan"))
        asm.assemble_matrix(a, A, bcs=bcs, diagonal=2.5)  # by default the walk
        asm.assemble_matrix(a, R, bcs=bcs, diagonal=2.5, variant=other)
        assert bool(((A.values - R.values).abs() <= tol).all())
        if bcs:
            masked = mark[row] | mark[col]
            assert torch.equal(A.values[masked], R.values[masked])
    asm.assemble_matrix(a, R, bcs=bcs, diagonal=2.5, variant="row-walk")
    assert torch.equal(A.values, R.values)  # "auto" is the walk, and a fixed order


@pytest.mark.parametrize("kind,n", [("p1", 2), ("p1k", 5), ("p2", 2), ("p2", 5), ("p3", 2), ("p3", 4), ("vp2", 2), ("vp2", 4)])
def test_walks_match_the_oracle(kind, n):
    P = fo.build_problem(kind, n, seed=n)
    R = run_system(P, variant="row-walk", precision="fp32" if kind == "vp2" else "fp64")
    ref = fo.solve_system(P)
    assert np.array_equal(R["row_ptr"], ref["row_ptr"]) and np.array_equal(R["col"], ref["col"])
    if kind == "vp2":  # FP32 element tensors
        assert np.linalg.norm(R["A"] - ref["A"]) < 2e-6 * np.linalg.norm(ref["A"])
        return
    ok, worst = tolerance_check(R["A"], ref["A"], ref["A_bound"])
    assert ok, worst
