"""Coefficients of a form given as FFCx bodies: the values of the call are the
host array's when the call returns, page-locked or not, however much work the
stream has before it."""
import numpy as np
import pytest

import ffcx_bodies as fb
from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("n", [2, 12])
def test_values_written_after_the_call_are_not_read(n, pinned):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    mesh = fem.create_unit_cube(n, jitter=0.2, seed=1)
    V, W = fem.functionspace(mesh, ("P", 2)), fem.functionspace(mesh, ("P", 1))
    k = fem.Function(W)
    keep = torch.empty(W.num_nodes, dtype=torch.float64, pin_memory=pinned)
    k.x.array = keep.numpy()
    old, new = np.random.default_rng(n).uniform(0.5, 2.0, (2, W.num_nodes))
    k.x.array[:] = old
    B = fb.stiffness(2, "p1")
    a = cx.form(fem.FFCxForm([fem.FFCxIntegral(B["integral_type"], B["name"], B["body"])], [V, V], [k]))
    asm = cx.CUDAAssembler()
    A, R = asm.create_matrix(a), asm.create_matrix(a)
    asm.assemble_matrix(a, R)
    torch.cuda.synchronize()
    scale = float(R.values.abs().max())
    for _ in range(2):
        torch.cuda._sleep(50_000_000)  # some 25 ms of the stream
        asm.assemble_matrix(a, A)
        k.x.array[:] = new
        torch.cuda.synchronize()
        # the same additions in another order
        assert float((A.values - R.values).abs().max()) <= 1e-13 * scale
        k.x.array[:] = old
