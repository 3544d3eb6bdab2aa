"""Vector-P2 row walk where nodes have empty rows (nodes of no cell, the padding
of the last group of three) and where the value array begins at an 8-byte but
not 16-byte aligned address: nothing outside the rows is written.  Compared
with the warp-coalesced scatter under the bound of test_gpu_rows_vp2.py; the
entries around the array keep their marks, bit for bit."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu

MARK = -7.25


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n,cells", [(1, [0]), (1, [0, 2]), (1, [0, 4]), (1, [0, 1, 2, 3, 4, 5]), (2, range(6)), (2, range(48)), (3, range(0, 162, 7)),
                                     (6, range(500, 1000))])
def test_empty_rows_and_unaligned_values(n, cells, offset):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem
    from cudolfinx.la import CUDAMatrix

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    mesh = fem.Mesh(m.geometry_x, m.cells[list(cells)], grid_n=n)
    V = fem.functionspace(mesh, ("P", 2, (3,)))
    a = cx.form(fem.elasticity(V, 1.25, 0.8, precision="fp32"))
    asm = cx.CUDAAssembler()
    R = asm.create_matrix(a)
    nnz = R.sparsity.nnz
    buf = torch.full((nnz + 8,), MARK, dtype=torch.float64, device="cuda")
    A = CUDAMatrix(R._ctx, R.sparsity, buf[2 + offset:2 + offset + nnz])
    rp, col = R.sparsity.to_host()
    N = len(rp) - 1
    row = np.repeat(np.arange(N), np.diff(rp))
    tol = None
    for dofs in ([], fem.locate_boundary_dofs(V)[::5]):
        bcs = asm.pack_bcs([fem.dirichletbc(0.0, dofs, V)] if len(dofs) else [])
        buf.fill_(MARK)
        asm.assemble_matrix(a, A, bcs=bcs, variant="row-walk")
        asm.assemble_matrix(a, R, bcs=bcs, variant="coalesced")
        got, ref, all_ = A.values.cpu().numpy(), R.values.cpu().numpy(), buf.cpu().numpy()
        if tol is None:
            d = np.zeros(N)
            d[row[row == col]] = ref[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max()
        assert np.all(np.abs(got - ref) <= tol)
        assert np.all(all_[:2 + offset] == MARK) and np.all(all_[2 + offset + nnz:] == MARK)
