"""P2 lifting without element tensors (FP64 forms): against the oracle's
element matrices, within its per-entry bound (rtol 1e-12 of the row's
|A_ij d_j| plus 1e-14 of the cell's largest entry times sum |d_j|; the two
4 x 4 products add some 60 terms of at most 16 times that entry at 2^-53,
below both parts together)."""
import numpy as np
import pytest

from conftest import ensure_library
from gpu_util import tolerance_check
from oracle import fem_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coef", ["const", "dg0", "p1"])
@pytest.mark.parametrize("n,dofs", [(1, "all"), (2, "one"), (3, "edges"), (5, "every third"), (6, "boundary")])
def test_p2_lifting_matches_oracle(n, dofs, coef):
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    rng = np.random.default_rng(n)
    # cells in any order, each with its vertices in any order (either orientation)
    mesh = fem.Mesh(m.geometry_x, rng.permuted(m.cells[rng.permutation(len(m.cells))], axis=1), grid_n=n)
    V = fem.functionspace(mesh, ("P", 2))
    kv = np.exp(rng.standard_normal(mesh.num_vertices))
    kc = np.exp(rng.standard_normal(mesh.num_cells))
    if coef == "const":
        k, kcell = 0.7, np.full((mesh.num_cells, 4), 0.7)
    elif coef == "dg0":
        k, kcell = fem.Function(fem.functionspace(mesh, ("DG", 0)), kc), np.repeat(kc[:, None], 4, axis=1)
    else:
        k, kcell = fem.Function(fem.functionspace(mesh, ("P", 1)), kv), kv[mesh.cells]
    sel = {"all": np.arange(V.num_dofs), "one": np.array([V.num_dofs // 2]), "edges": np.unique(V.dofs[:, 4:]),
           "every third": np.arange(0, V.num_dofs, 3), "boundary": fem.locate_boundary_dofs(V)}[dofs]
    g, x0, b0 = rng.standard_normal((3, V.num_dofs))
    asm = cx.CUDAAssembler()
    a = cx.form(fem.stiffness(V, k))
    bcs = asm.pack_bcs([fem.dirichletbc(fem.Function(V, g), sel.astype(np.int32))])
    marker = np.zeros(V.num_dofs, dtype=np.uint8)
    marker[sel] = 1
    Ae = fo.p2_stiffness(mesh.geometry_x, mesh.cells, kcell)
    L = cx.form(fem.load(V, 0.0))
    b = asm.assemble_vector(L)
    x = asm.assemble_vector(L)
    for shift, scale in ((None, 1.0), (x0, -0.75)):
        b.vector.copy_(_like(b, b0))
        if shift is not None:
            x.vector.copy_(_like(x, shift))
        asm.apply_lifting(b, [a], [bcs], x0=None if shift is None else [x], scale=scale)
        ref = fo.apply_lifting(b0.copy(), Ae, V.dofs, V.dofs, marker, g, shift, scale)
        bound = fo.lifting_bound(V.num_dofs, Ae, V.dofs, V.dofs, marker, g, shift, scale) + fo.PARITY_RTOL * np.abs(b0)
        ok, worst = tolerance_check(b.to_host(), ref, bound)
        assert ok, worst


def _like(b, v):
    import torch

    return torch.as_tensor(v, device=b.vector.device)
