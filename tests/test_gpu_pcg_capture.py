"""The FP64 solver under stream capture: refused before it enqueues anything, so
that the capture holds what came before and after it and nothing of the solve."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


def test_solve_is_refused_and_leaves_nothing_in_the_graph():
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    V = fem.functionspace(fem.create_unit_cube(3), ("P", 1))
    asm = cx.CUDAAssembler()
    a, L = cx.form(fem.stiffness(V, 1.0)), cx.form(fem.load(V, 1.0))
    bc = fem.dirichletbc(0.0, fem.locate_boundary_dofs(V), V)
    A, b = asm.assemble_matrix(a, bcs=[bc]), asm.assemble_vector(L)
    asm.set_bc(b, [bc], V)
    x, its, _ = asm.solve(A, b, rtol=1e-10)
    want = x.to_host()
    y = torch.zeros(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y += 1.0
        with pytest.raises(RuntimeError, match="cannot be captured"):
            asm.solve(A, b, x, rtol=1e-10)
        y += 1.0
    x.vector.fill_(3.0)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), np.full(4, 2.0)) and np.all(x.to_host() == 3.0)
    again, its2, _ = asm.solve(A, b, rtol=1e-10)
    assert its == its2 and np.array_equal(again.to_host(), want)
