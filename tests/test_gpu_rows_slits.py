"""The P2 / P3 row walk on dofmaps with slits: neighbouring cells that share some
of the dofs of their common face and have their own for the others.  A walk
around an edge carries sums from a cell to the next one across that face, so
it has to be refused where the two cells do not name the same dofs; where it is
accepted it has to agree with the thread-per-cell scatter under the bound of
test_gpu_rows.py."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


def _space(mesh, degree, split):
    """A P2 / P3 space in which `split` = [(cell, its local dofs with numbers of their own)]."""
    from cudolfinx import fem

    V = fem.functionspace(mesh, ("P", degree))
    for c, local in split:
        V.dofs[c, local] = V.num_nodes + np.arange(len(local))
        V.num_nodes += len(local)
    return V


def _matches(V, k, variant):
    import cudolfinx as cx
    from cudolfinx import fem

    a = cx.form(fem.stiffness(V, k))
    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    rp, col = A.sparsity.to_host()
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    A.values.fill_(float("nan"))
    asm.assemble_matrix(a, A, variant=variant)
    asm.assemble_matrix(a, R, variant="atomic-full")
    got, ref = A.values.cpu().numpy(), R.values.cpu().numpy()
    d = np.zeros(len(rp) - 1)
    d[row[row == col]] = ref[row == col]
    return np.all(np.abs(got - ref) <= 1e-12 * np.sqrt(d[row] * d[col]) + 1e-14 * np.abs(ref).max())


def _mesh(cells):
    from cudolfinx import fem

    m = fem.create_unit_cube(1, jitter=0.2, seed=4)
    return fem.Mesh(m.geometry_x, m.cells[list(cells)], grid_n=1)


@pytest.mark.parametrize("cells", [[0, 1], [0, 2], [0, 1, 3], range(6)])
@pytest.mark.parametrize("degree", [2, 3])
def test_slits(degree, cells):
    ensure_library()
    mesh = _mesh(cells)
    base = _space(mesh, degree, []).dofs.copy()
    refused = 0
    for seed in range(25):
        rng = np.random.default_rng(seed)
        c = int(rng.integers(mesh.num_cells))
        # local dofs of cell c that other cells have too: a random part of them becomes its own
        shared = [q for q in range(base.shape[1]) if np.any(np.delete(base, c, axis=0) == base[c, q])]
        own = [q for q in shared if rng.random() < rng.choice([0.15, 0.5, 0.85])]
        V = _space(mesh, degree, [(c, own)])
        k = float(rng.uniform(0.5, 2.0))
        assert _matches(V, k, "auto")
        try:
            ok = _matches(V, k, "row-walk")
        except RuntimeError as e:
            assert "row walk" in str(e)
            refused += 1
            continue
        assert ok, (seed, c, own)
    assert refused > 0


@pytest.mark.parametrize("degree", [2, 3])
def test_slit_that_ends_at_an_edge(degree):
    """Two cells with a common face share the dofs of one of its edges and have
    their own for its third vertex and that vertex's edges."""
    ensure_library()
    mesh = _mesh([0, 1])
    u, v, w = sorted(set(mesh.cells[0]) & set(mesh.cells[1]))
    V = _space(mesh, degree, [])
    one = list(mesh.cells[1])
    edges = ((2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1))
    local = [one.index(w)]
    for e, ends in enumerate(edges):
        if {one[ends[0]], one[ends[1]]} in ({u, w}, {v, w}):
            local += [4 + (degree - 1) * e + s for s in range(degree - 1)]
    if degree == 3:
        local.append(16 + next(q for q in range(4) if one[q] not in (u, v, w)))
    V = _space(mesh, degree, [(1, local)])
    assert _matches(V, 0.7, "auto")
    with pytest.raises(RuntimeError, match="row walk"):
        _matches(V, 0.7, "row-walk")
