"""AssemblyGraph where the row walk wins a size class and a later mesh of the class
cannot take it: that mesh goes on with the scatter.  Two P3 meshes of one
class, the second with a cell listed twice (which the P3 walk does not take);
the timings are replaced so that the last candidate wins.  Bound: that of
test_gpu_rows.py."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


def test_a_class_whose_later_mesh_has_no_walk(monkeypatch):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(2, jitter=0.2, seed=5)
    asm = cx.CUDAAssembler()
    items = []
    for cells in (np.arange(48), np.append(np.arange(48), 7)):
        V = fem.functionspace(fem.Mesh(m.geometry_x, m.cells[cells], grid_n=2), ("P", 3))
        a = cx.form(fem.stiffness(V, 0.7))
        items.append((a, asm.create_matrix(a), [fem.dirichletbc(0.0, fem.locate_boundary_dofs(V)[::3], V)]))
    ticks = iter(range(10 ** 6))
    monkeypatch.setattr(torch.cuda.Event, "elapsed_time", lambda self, end: 1.0 / (1 + next(ticks)))
    g = cx.AssemblyGraph(items)
    assert len(g.tuner.cache) == 1  # one class
    for _, A, _ in items:
        A.values.fill_(float("nan"))
    g.capture().replay()
    for a, A, bcs in items:
        got = A.values.cpu().numpy()
        R = asm.create_matrix(a)
        asm.assemble_matrix(a, R, variant="atomic-full")
        rp, col = R.sparsity.to_host()
        row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        ref = R.values.cpu().numpy()
        d = np.zeros(len(rp) - 1)
        d[row[row == col]] = ref[row == col]
        tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max()
        asm.assemble_matrix(a, R, bcs=bcs, variant="atomic-full")
        assert np.all(np.abs(got - R.values.cpu().numpy()) <= tol)
