"""Matrices of forms given as FFCx bodies at the edges of the 32-entity tiles
(one cell, 31..33 cells, several tiles with a remainder), against the built-in
kernel of the same form.  Element matrices are positive semi-definite, so an
entry's |contributions| sum to at most sqrt(A_ii A_jj); the two evaluations
differ by their rounding (below 1e-13 of an element's entries) and the order
of the sums: 1e-12 of that bound."""
import numpy as np
import pytest

import ffcx_bodies as fb
from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("degree", [1, 2])
def test_tile_edges(degree, cells):
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    full = fem.create_unit_cube(3, jitter=0.2, seed=2)
    mesh = fem.Mesh(full.geometry_x, full.cells[:cells], grid_n=3)
    V = fem.functionspace(mesh, ("P", degree))
    k = fem.Function(fem.functionspace(mesh, ("DG", 0)), np.exp(np.random.default_rng(3).standard_normal(cells)))
    B = fb.stiffness(degree, "dg0")
    a = cx.form(fem.FFCxForm([fem.FFCxIntegral(B["integral_type"], B["name"], B["body"])], [V, V], [k]))
    ref = cx.form(fem.stiffness(V, k))
    bc = fem.dirichletbc(0.0, fem.locate_boundary_dofs(V)[::3], V)
    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(ref)
    rp, col, _ = A.device_csr()
    rp, col = rp.cpu().numpy(), col.cpu().numpy()
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    tol = None
    for bcs in ([], [bc]):
        A.values.fill_(float("nan"))
        asm.assemble_matrix(a, A, bcs=bcs, diagonal=1.5)
        asm.assemble_matrix(ref, R, bcs=bcs, diagonal=1.5, variant="atomic-full")
        got, want = A.values.cpu().numpy(), R.values.cpu().numpy()
        if tol is None:
            d = np.zeros(V.num_dofs)
            d[row[row == col]] = want[row == col]
            tol = 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(want).max()
        assert np.all(np.abs(got - want) <= tol)


def test_tables_move_to_constant_memory_only_when_literal():
    """Tables of literals at a cell body's top level become file-scope
    constant data; others, and a facet body's, stay where they are."""
    ensure_library()
    import ctypes

    from cudolfinx import _lib

    def source(itype, body):
        n = ctypes.c_int64()
        args = (itype, 2, 4, 1, 4, 1, 0, None, b"tabulate_x", body.encode())
        _lib.check(_lib.lib.fe_ffcx_source(*args, None, 0, ctypes.byref(n)))
        buf = ctypes.create_string_buffer(n.value + 1)
        _lib.check(_lib.lib.fe_ffcx_source(*args, buf, n.value + 1, ctypes.byref(n)))
        return buf.value.decode()

    table = "alignas(32) static const double T[2][2] = {{1.0, -2.5e-3}, {0.0, 4}};\n"
    use = "for (int i = 0; i < 2; ++i) A[i] += T[i][0];\n"
    assert "static __constant__ double T[2][2]" in source(0, table + use)
    assert "__constant__" not in source(1, table + use)  # indexed by facet: lanes differ
    for kept in ("static const double T[2][2] = {{1.0, one}, {0.0, 4}};\n",
                 "{ static const double T[2][2] = {{1.0, 2.0}, {0.0, 4}}; A[0] += T[0][0]; }\n",
                 "// static const double T[2][2] = {{1.0, 2.0}, {0.0, 4}};\n",
                 "static const double T[9000] = {1.0};\n"):
        assert "__constant__" not in source(0, kept)
