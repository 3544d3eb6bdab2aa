"""FP32 element tensors in AssemblyGraph: the matrix does not depend on what the
tuner measures.  Variants that round an entry alike add the same FP32 numbers in
FP64, some tens of terms (24 cells, nine component blocks for a node-block
diagonal) of at most sqrt(A_ii A_jj) each: another order moves an entry by less
than 1e-13 of the largest one.  Variants that round differently are 3e-9 to 5e-8
apart."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,coef,n", [("p2", "dg0", 2), ("p2", "dg0", 15), ("p2", "dg0", 16), ("p2", "dg0", 22), ("p2", "p1", 3),
                                         ("p2", "p1", 17), ("vp2", "dg0", 2), ("vp2", "dg0", 17), ("vp2", "dg0", 19)])
def test_timings_do_not_decide_values(kind, coef, n, monkeypatch):
    ensure_library()
    import torch

    import cudolfinx as cx
    from cudolfinx import fem

    mesh = fem.create_unit_cube(n, jitter=0.2, seed=n)
    rng = np.random.default_rng(n)
    Q = fem.functionspace(mesh, ("DG", 0) if coef == "dg0" else ("P", 1))
    k, mu = (fem.Function(Q, np.exp(rng.standard_normal(Q.num_nodes))) for _ in range(2))
    if kind == "p2":
        a = cx.form(fem.stiffness(fem.functionspace(mesh, ("P", 2)), k, precision="fp32"))
    else:
        a = cx.form(fem.elasticity(fem.functionspace(mesh, ("P", 2, (3,))), k, mu, precision="fp32"))
    A = cx.CUDAAssembler().create_matrix(a)
    monkeypatch.setattr(torch.cuda.Event, "elapsed_time", lambda self, end: float(rng.random()))
    first = None
    for _ in range(12):
        A.values.fill_(float("nan"))
        cx.AssemblyGraph([(a, A, [])]).run_eager()
        got = A.values.cpu().numpy()
        if first is None:
            first = got
        assert np.max(np.abs(got - first)) <= 1e-13 * np.abs(first).max()
