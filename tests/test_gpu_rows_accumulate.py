"""Calls that add to a matrix (zero=False) on several streams at once: no
addition is lost, with the row walk as with the scatter.  Every call adds the
same rows, so after `calls` of them on a zeroed matrix an entry is `calls` times
the single call's, to the rounding of `calls` additions."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("p1", 33), ("p2", 23), ("p3", 12), ("vp2", 12)])
def test_concurrent_additions(kind, n):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    mesh = fem.create_unit_cube(n, jitter=0.2, seed=1)
    V = fem.functionspace(mesh, {"p1": ("P", 1), "p2": ("P", 2), "p3": ("P", 3), "vp2": ("P", 2, (3,))}[kind])
    asm = cx.CUDAAssembler()
    streams = [torch.cuda.Stream() for _ in range(4)]
    forms = [cx.form(fem.elasticity(V, 1.0, 0.5, precision="fp32") if kind == "vp2" else fem.stiffness(V, 0.7))
             for _ in streams]
    A, R = asm.create_matrix(forms[0]), asm.create_matrix(forms[0])
    bcs = asm.pack_bcs([fem.dirichletbc(0.0, fem.locate_boundary_dofs(V)[::2], V)])
    for a in forms:  # plans and BC tables
        asm.assemble_matrix(a, R, bcs=bcs, variant="row-walk")
    A.values.zero_()
    torch.cuda.synchronize()
    rounds = 6
    for _ in range(rounds):
        for a, st in zip(forms, streams):
            with torch.cuda.stream(st):
                asm.assemble_matrix(a, A, bcs=bcs, zero=False, variant="row-walk")
    torch.cuda.synchronize()
    got, one = A.values.cpu().numpy(), R.values.cpu().numpy()
    calls = rounds * len(forms)
    rp, col = A.sparsity.to_host()
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    mark = np.zeros(len(rp) - 1, dtype=bool)
    mark[fem.locate_boundary_dofs(V)[::2]] = True
    want = np.where((row == col) & mark[row], one, calls * one)  # the BC rows' diagonal is set, not added
    assert np.all(np.abs(got - want) <= calls * calls * 2.0 ** -52 * np.abs(one))
