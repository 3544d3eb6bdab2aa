"""The row walk (variant "row-walk", the default of large FP64 P1 / P2 / P3 matrices) against
the thread-per-cell scatter into both triangles (variant "atomic-full").

The element matrices are positive semi-definite, so the sum of an entry's
|contributions| is at most sqrt(A_ii A_jj) (Cauchy-Schwarz over the cells):
the two summation orders differ by less than 1e-12 of it (some tens of terms
at 2^-53), and an element's own rounding is below 1e-14 of the largest entry.
"""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu

SPACE = {"p1": ("P", 1), "p2": ("P", 2), "p3": ("P", 3)}


def _mesh(n, order, seed=0, cells=None):
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=seed)
    c = m.cells if cells is None else m.cells[np.asarray(cells)]
    if order == "permuted":  # cells in any order, each with its vertices in any order
        rng = np.random.default_rng(seed)
        c = rng.permuted(c[rng.permutation(len(c))], axis=1)
    return fem.Mesh(m.geometry_x, c, grid_n=n)


def _form(kind, coef, mesh, seed=1):
    import cudolfinx as cx
    from cudolfinx import fem

    V = fem.functionspace(mesh, SPACE[kind])
    rng = np.random.default_rng(seed)
    if coef == "const":
        k = 0.7
    elif coef == "dg0":
        k = fem.Function(fem.functionspace(mesh, ("DG", 0)), np.exp(rng.standard_normal(mesh.num_cells)))
    else:
        k = fem.Function(fem.functionspace(mesh, ("P", 1)), np.exp(rng.standard_normal(mesh.num_vertices)))
    return V, cx.form(fem.stiffness(V, k))


def _structure(A):
    rp, col, _ = A.device_csr()
    rp, col = rp.cpu().numpy(), col.cpu().numpy()
    return np.repeat(np.arange(len(rp) - 1), np.diff(rp)), col


def _compare(V, a, bcs, diagonal=1.0, variant="row-walk"):
    """The walk's matrix against the scatter's, without BCs and with them; a
    repeated call (bitwise equal for the walk) and one that adds."""
    import cudolfinx as cx

    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    row, col = _structure(A)
    tol = None
    for b in ([], bcs):
        c = asm.pack_bcs(b)
        A.values.fill_(float("nan"))
        asm.assemble_matrix(a, A, bcs=c, diagonal=diagonal, variant=variant)
        asm.assemble_matrix(a, R, bcs=c, diagonal=diagonal, variant="atomic-full")
        A.assemble()
        got, ref = A.values.cpu().numpy(), R.values.cpu().numpy()
        if tol is None:  # from the unmasked matrix
            d = np.zeros(V.num_dofs)
            d[row[row == col]] = ref[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * (np.abs(ref).max() if ref.size else 0.0)
        mark = np.zeros(V.num_dofs, dtype=bool)
        for q in b:
            mark[q.dofs] = True
        masked = mark[row] | mark[col]
        assert np.all(np.abs(got - ref)[~masked] <= tol[~masked])
        assert np.array_equal(got[masked], np.where((row == col) & mark[row], diagonal, 0.0)[masked])
    asm.assemble_matrix(a, A, bcs=c, diagonal=diagonal, variant=variant)
    again = A.values.cpu().numpy()
    if variant == "row-walk":
        assert np.array_equal(again, got)
    asm.assemble_matrix(a, A, bcs=c, diagonal=diagonal, zero=False, variant=variant)
    want = np.where(masked, again, 2.0 * again)
    assert np.all(np.abs(A.values.cpu().numpy() - want) <= 2.0 * np.where(masked, 0.0, tol))


@pytest.mark.parametrize("order", ["natural", "permuted"])
@pytest.mark.parametrize("coef", ["const", "dg0", "p1"])
@pytest.mark.parametrize("kind,n", [("p1", 1), ("p1", 3), ("p1", 10), ("p2", 1), ("p2", 2), ("p2", 7), ("p1", 33), ("p2", 23),
                                    ("p3", 1), ("p3", 2), ("p3", 5)])
def test_walk_matches_scatter(kind, n, coef, order):
    ensure_library()
    if kind == "p3" and coef == "p1":
        pytest.skip("P3 stiffness takes a constant or cellwise coefficient")
    from cudolfinx import fem

    mesh = _mesh(n, order, seed=n)
    V, a = _form(kind, coef, mesh)
    bc = fem.dirichletbc(0.0, fem.locate_boundary_dofs(V)[::2], V)  # every other boundary dof
    _compare(V, a, [bc], diagonal=2.5)


@pytest.mark.parametrize("cells", [[0], [0, 3], [0, 1, 3, 4], [5, 4, 2, 0], [0, 1, 2, 3, 4]])
@pytest.mark.parametrize("kind", ["p1", "p2", "p3"])
def test_open_and_separate_fans(kind, cells):
    """Some of the six cells around the cube's diagonal: one cell, cells that
    share only an edge (two fans), open fans; nodes of no cell."""
    ensure_library()
    from cudolfinx import fem

    mesh = _mesh(1, "natural", cells=cells)
    V, a = _form(kind, "dg0" if kind == "p3" else "p1", mesh)
    _compare(V, a, [fem.dirichletbc(0.0, np.array([0, V.num_dofs - 1]), V)])


@pytest.mark.parametrize("kind", ["p1", "p2", "p3"])
def test_overlapping_cells(kind):
    """Cells listed twice: a vertex row adds them all; a walk around an edge
    writes each slot once, so P2 and P3 refuse them and "auto" takes the scatter."""
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    mesh = _mesh(2, "natural", cells=list(range(48)) + [7, 7, 20])
    V, a = _form(kind, "dg0", mesh)
    _compare(V, a, [fem.dirichletbc(0.0, fem.locate_boundary_dofs(V), V)],
             variant="row-walk" if kind == "p1" else "auto")
    if kind != "p1":
        with pytest.raises(RuntimeError, match="row walk"):
            cx.CUDAAssembler().assemble_matrix(a, variant="row-walk")


@pytest.mark.parametrize("kind", ["p1", "p2", "p3"])
def test_pattern_with_more_slots(kind):
    """A pattern with couplings the form does not have: their slots are zero."""
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import _lib, fem
    from cudolfinx.la import CUDAMatrix, Sparsity

    mesh = _mesh(3, "natural")
    V, a = _form(kind, "const", mesh)
    asm = cx.CUDAAssembler()
    A = asm.create_matrix(a)
    rp, col, _ = A.device_csr()
    rp, col = rp.cpu().numpy(), col.cpu().numpy()
    N = len(rp) - 1
    wide = [np.union1d(col[rp[r]:rp[r + 1]], [0, r // 2, N - 1]).astype(np.int32) for r in range(N)]
    rp2 = np.concatenate([[0], np.cumsum([len(w) for w in wide])]).astype(np.int32)
    col2 = np.concatenate(wide)
    ctx = cx.get_cuda_context()
    h = _lib.out_handle()
    _lib.check(_lib.lib.fe_sparsity_create(ctx.handle, rp2.ctypes.data, col2.ctypes.data, N, N, h))
    B = CUDAMatrix(ctx, Sparsity(ctx, h.value))
    B.values.fill_(float("nan"))
    V2, a2 = _form(kind, "const", mesh)
    asm.assemble_matrix(a, A, variant="row-walk")
    asm.assemble_matrix(a2, B, variant="row-walk")
    B.assemble()
    want = np.zeros(len(col2))
    vals = A.values.cpu().numpy()
    for r in range(N):
        want[rp2[r] + np.searchsorted(wide[r], col[rp[r]:rp[r + 1]])] = vals[rp[r]:rp[r + 1]]
    assert np.array_equal(B.values.cpu().numpy(), want)


@pytest.mark.parametrize("kind,n", [("p1", 33), ("p2", 23)])
def test_large_meshes_walk_by_default(kind, n):
    """From the size on, "auto" is the walk, bit for bit; two BC collections
    on rows and columns, FP32 element tensors and a coefficient in another
    numbering go on with the scatter."""
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    mesh = _mesh(n, "natural")
    V, a = _form(kind, "p1", mesh)
    asm = cx.CUDAAssembler()
    A, B = asm.create_matrix(a), asm.create_matrix(a)
    asm.assemble_matrix(a, A)
    asm.assemble_matrix(a, B, variant="row-walk")
    assert np.array_equal(A.values.cpu().numpy(), B.values.cpu().numpy())
    if kind == "p2":
        b = cx.form(fem.stiffness(V, a._spec.coefficients[0], precision="fp32"))
        asm.assemble_matrix(b, B)
        d = np.linalg.norm(B.values.cpu().numpy() - A.values.cpu().numpy())
        assert 0.0 < d < 2e-6 * np.linalg.norm(A.values.cpu().numpy())
    k = fem.Function(fem.functionspace(mesh, ("DG", 1)))  # four values a cell: not the vertices' numbering
    k.x.array[:] = a._spec.coefficients[0].x.array[mesh.cells.ravel()]
    c = cx.form(fem.stiffness(V, k))
    asm.assemble_matrix(c, B)
    ref = A.values.cpu().numpy()
    assert np.max(np.abs(B.values.cpu().numpy() - ref)) <= 1e-13 * np.abs(ref).max()
