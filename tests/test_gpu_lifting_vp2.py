"""Vector-P2 elasticity lifting without element tensors (FP64 forms): against
the oracle's element matrices, within its per-entry bound (rtol 1e-12 of the
row's |A_ij d_j| plus 1e-14 of the cell's largest entry times sum |d_j|; the
stresses and their products with the gradients add some 100 terms of at most
16 times that entry at 2^-53, below both parts together)."""
import numpy as np
import pytest

from conftest import ensure_library
from gpu_util import tolerance_check
from oracle import fem_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coef", ["const", "dg0"])
@pytest.mark.parametrize("n,dofs", [(1, "all"), (2, "one"), (3, "edges"), (4, "every seventh"), (5, "boundary")])
def test_vp2_lifting_matches_oracle(n, dofs, coef):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    m = fem.create_unit_cube(n, jitter=0.2, seed=n)
    rng = np.random.default_rng(n)
    # cells in any order, each with its vertices in any order (either orientation)
    mesh = fem.Mesh(m.geometry_x, rng.permuted(m.cells[rng.permutation(len(m.cells))], axis=1), grid_n=n)
    V = fem.functionspace(mesh, ("P", 2, (3,)))
    if coef == "const":
        lam, mu, lc, mc = 1.25, 0.8, np.full(mesh.num_cells, 1.25), np.full(mesh.num_cells, 0.8)
    else:
        Q = fem.functionspace(mesh, ("DG", 0))
        lc, mc = np.exp(rng.standard_normal((2, mesh.num_cells)))
        lam, mu = fem.Function(Q, lc), fem.Function(Q, mc)
    sel = {"all": np.arange(V.num_dofs), "one": np.array([V.num_dofs // 2]),
           "edges": (3 * np.unique(V.dofs[:, 4:])[:, None] + np.arange(3)).ravel(),
           "every seventh": np.arange(0, V.num_dofs, 7), "boundary": fem.locate_boundary_dofs(V)}[dofs]
    g, x0, b0 = rng.standard_normal((3, V.num_dofs))
    asm = cx.CUDAAssembler()
    a = cx.form(fem.elasticity(V, lam, mu))
    bcs = asm.pack_bcs([fem.dirichletbc(fem.Function(V, g), sel.astype(np.int32))])
    marker = np.zeros(V.num_dofs, dtype=np.uint8)
    marker[sel] = 1
    Ae = fo.p2_elasticity(mesh.geometry_x, mesh.cells, lc, mc)
    L = cx.form(fem.load(V, (0.0, 0.0, 0.0)))
    b, x = asm.assemble_vector(L), asm.assemble_vector(L)
    for shift, scale in ((None, 1.0), (x0, -0.75)):
        b.vector.copy_(torch.as_tensor(b0))
        if shift is not None:
            x.vector.copy_(torch.as_tensor(shift))
        asm.apply_lifting(b, [a], [bcs], x0=None if shift is None else [x], scale=scale)
        ref = fo.apply_lifting(b0.copy(), Ae, V.dofs, V.dofs, marker, g, shift, scale, 3, 3)
        bound = fo.lifting_bound(V.num_dofs, Ae, V.dofs, V.dofs, marker, g, shift, scale, 3, 3)
        ok, worst = tolerance_check(b.to_host(), ref, bound + fo.PARITY_RTOL * np.abs(b0))
        assert ok, worst
