"""The warp-coalesced vector-P2 scatter at its three walk lengths (4, 8 and 16
cells a warp): against the thread-per-cell scatter into both triangles
(variant "atomic-full"), FP64 element tensors.

An entry's sum of |contributions| is at most a small multiple of
sqrt(A_ii A_jj); some tens of terms in another order differ by less than
1e-12 of it, and an element's own rounding is below 1e-14 of the largest entry.
"""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cells", [(1, 1), (1, 5), (2, 48), (9, 4374), (10, 4736), (10, 4737), (10, 4741), (12, 10368),
                                     (28, 131071), (28, 131072), (28, 131705)])
def test_walk_lengths(n, cells):
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    mesh = fem.Mesh(m.geometry_x, m.cells[:cells], grid_n=n)  # the last warp's walk ends early
    V = fem.functionspace(mesh, ("P", 2, (3,)))
    Q = fem.functionspace(mesh, ("DG", 0))
    rng = np.random.default_rng(n)
    lam, mu = (fem.Function(Q, np.exp(rng.standard_normal(cells))) for _ in range(2))
    asm = cx.CUDAAssembler()
    a = cx.form(fem.elasticity(V, lam, mu))
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    dofs = np.arange(0, V.num_dofs, 7, dtype=np.int32)
    for bcs in ([], [fem.dirichletbc(0.0, dofs, V)]):
        c = asm.pack_bcs(bcs)
        asm.assemble_matrix(a, A, bcs=c, variant="coalesced")
        asm.assemble_matrix(a, R, bcs=c, variant="atomic-full")
        got, ref = A.values.cpu().numpy(), R.values.cpu().numpy()
        if not bcs:
            rp, col, _ = A.device_csr()
            rp, col = rp.cpu().numpy(), col.cpu().numpy()
            row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
            d = np.zeros(len(rp) - 1)
            d[row[row == col]] = ref[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max()
        assert np.all(np.abs(got - ref) <= tol)
