"""The row walk on patterns of the caller's own, with nodes of no cell: their rows
hold other columns left and right of the diagonal, only the diagonal, or none at
all.  A BC row's diagonal value stands at the row's own column, as the scatter
puts it; the bound is that of test_gpu_rows.py (test_gpu_rows_vp2.py for FP32
vector P2)."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu

SPACE = {"p1": ("P", 1), "p2": ("P", 2), "p3": ("P", 3), "vp2": ("P", 2, (3,))}


def _pattern(V, extra):
    """Block columns of every node: its cells' nodes, and extra(r) for a node of no cell."""
    cols = [set() for _ in range(V.num_nodes)]
    for d in V.dofs:
        for r in d:
            cols[r].update(d.tolist())
    return [sorted(c if c else set(extra(r)) & set(range(V.num_nodes))) for r, c in enumerate(cols)]


@pytest.mark.parametrize("extra", ["left", "diagonal", "none", "without diagonal"])
@pytest.mark.parametrize("kind", ["p1", "p2", "p3", "vp2"])
def test_nodes_of_no_cell(kind, extra):
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem
    from cudolfinx.la import CUDAMatrix, Sparsity

    m = fem.create_unit_cube(2, jitter=0.2, seed=2)
    mesh = fem.Mesh(m.geometry_x, m.cells[[0, 7, 8, 20, 21]], grid_n=2)
    V = fem.functionspace(mesh, SPACE[kind])
    bs = V.bs
    a = cx.form(fem.elasticity(V, 1.25, 0.8, precision="fp32") if kind == "vp2" else fem.stiffness(V, 0.7))
    cols = _pattern(V, {"left": lambda r: (0, r // 2, r, r + 3), "diagonal": lambda r: (r,), "none": lambda r: (),
                        "without diagonal": lambda r: (r - 2, r + 1)}[extra])
    scalar = [[bs * c + q for c in cols[r // bs] for q in range(bs)] for r in range(bs * V.num_nodes)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in scalar])])
    col = np.concatenate([np.asarray(c, dtype=int) for c in scalar])
    ctx = cx.get_cuda_context()
    S = Sparsity.from_csr(ctx, rp, col, len(rp) - 1)
    A, R = CUDAMatrix(ctx, S), CUDAMatrix(ctx, S)
    asm = cx.CUDAAssembler()
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    dofs = np.arange(0, len(rp) - 1, 2, dtype=np.int32)
    for bcs in ([], [fem.dirichletbc(0.0, dofs, V)]):
        A.values.fill_(float("nan"))
        asm.assemble_matrix(a, R, bcs=bcs, diagonal=2.5, variant="coalesced" if kind == "vp2" else "atomic-full")
        try:
            asm.assemble_matrix(a, A, bcs=bcs, diagonal=2.5, variant="row-walk")
        except RuntimeError as e:
            # vector P2: a diagonal that is missing is left to the scatter
            assert kind == "vp2" and extra == "without diagonal" and "row walk" in str(e)
            asm.assemble_matrix(a, A, bcs=bcs, diagonal=2.5)
        got, ref = A.values.cpu().numpy(), R.values.cpu().numpy()
        if not bcs:
            d = np.zeros(len(rp) - 1)
            d[row[row == col]] = ref[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max()
            assert np.all(np.abs(got - ref) <= tol)
            continue
        mark = np.zeros(len(rp) - 1, dtype=bool)
        mark[dofs] = True
        masked = mark[row] | mark[col]
        assert np.array_equal(got[masked], np.where((row == col) & mark[row], 2.5, 0.0)[masked])
        assert np.array_equal(got[masked], ref[masked])
        assert np.all(np.abs(got - ref) <= tol)
