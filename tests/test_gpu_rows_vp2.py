"""The row walk of FP32 vector-P2 elasticity (variant "row-walk")
against the warp-coalesced scatter (variant "coalesced").

Both add the same element entries, rounded to FP32 alike, in FP64: an entry's
sum of |contributions| is at most a small multiple of sqrt(A_ii A_jj), and
some 200 terms (24 cells times nine blocks, for a node-block diagonal) at
2^-53 stay below 1e-12 of it.
"""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


def _form(n, order, coef, cells=None):
    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    c = m.cells if cells is None else m.cells[np.asarray(cells)]
    rng = np.random.default_rng(n)
    if order == "permuted":  # cells in any order, each with its vertices in any order
        c = rng.permuted(c[rng.permutation(len(c))], axis=1)
    mesh = fem.Mesh(m.geometry_x, c, grid_n=n)
    V = fem.functionspace(mesh, ("P", 2, (3,)))
    if coef == "const":
        lam, mu = 1.25, 0.8
    else:
        Q = fem.functionspace(mesh, ("DG", 0))
        lam, mu = (fem.Function(Q, np.exp(rng.standard_normal(mesh.num_cells))) for _ in range(2))
    return V, cx.form(fem.elasticity(V, lam, mu, precision="fp32"))


@pytest.mark.parametrize("coef", ["const", "dg0"])
@pytest.mark.parametrize("n,order,cells", [(1, "natural", None), (1, "natural", [0]), (1, "permuted", [0, 3]), (2, "permuted", None),
                                           (5, "natural", None), (5, "permuted", None), (9, "natural", None), (11, "natural", None)])
def test_walk_matches_scatter(n, order, cells, coef):
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    V, a = _form(n, order, coef, cells)
    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    rp, col, _ = A.device_csr()
    rp, col = rp.cpu().numpy(), col.cpu().numpy()
    N = len(rp) - 1
    row = np.repeat(np.arange(N), np.diff(rp))
    tol = None
    for dofs in ([], fem.locate_boundary_dofs(V)[::2]):
        c = asm.pack_bcs([fem.dirichletbc(0.0, dofs, V)] if len(dofs) else [])
        A.values.fill_(float("nan"))
        asm.assemble_matrix(a, A, bcs=c, diagonal=2.5, variant="row-walk")
        asm.assemble_matrix(a, R, bcs=c, diagonal=2.5, variant="coalesced")
        got, ref = A.values.cpu().numpy(), R.values.cpu().numpy()
        if tol is None:  # from the matrix without BCs
            d = np.zeros(N)
            d[row[row == col]] = ref[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max()
        mark = np.zeros(N, dtype=bool)
        mark[dofs] = True
        masked = mark[row] | mark[col]
        assert np.all(np.abs(got - ref)[~masked] <= tol[~masked])
        assert np.array_equal(got[masked], np.where((row == col) & mark[row], 2.5, 0.0)[masked])
    asm.assemble_matrix(a, A, bcs=c, diagonal=2.5, variant="row-walk")
    assert np.array_equal(A.values.cpu().numpy(), got)  # a fixed order
    asm.assemble_matrix(a, A, bcs=c, diagonal=2.5, zero=False, variant="row-walk")
    want = np.where(masked, got, 2.0 * got)
    assert np.all(np.abs(A.values.cpu().numpy() - want) <= np.where(masked, 0.0, 2.0 * tol))


def test_walk_is_not_offered_for_fp64_tensors():
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    mesh = fem.create_unit_cube(2)
    V = fem.functionspace(mesh, ("P", 2, (3,)))
    asm = cx.CUDAAssembler()
    with pytest.raises(RuntimeError, match="row walk"):
        asm.assemble_matrix(cx.form(fem.elasticity(V, 1.0, 1.0)), variant="row-walk")
