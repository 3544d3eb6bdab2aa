"""The FP64 solver on both sides of the lines between its two-kernel and its
five-launch iteration.  b = A x with a known x; the matrices are strictly
diagonally dominant by a factor of two, so their condition number is below 3
times the ratio of their diagonal entries (below 20), and rtol 1e-13 leaves an
error below 1e-11."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,band", [(280000, [1, 70, 4900]), (280001, [1, 70, 4900]),     # 7 a row: rows
                                    (39500, range(1, 41)), (39550, range(1, 41)),          # 81 a row: 3.2 M nonzeros
                                    (1200000, [1, 400]), (1199000, [1, 400]),              # 5 a row: 6 M nonzeros
                                    (222500, range(1, 14)), (221500, range(1, 14))])       # 27 a row: 6 M nonzeros
def test_both_sides(n, band):
    ensure_library()
    import scipy.sparse as sp
    import torch

    import cudolfinx as cx
    from cudolfinx.la import CUDAMatrix, CUDAVector, Sparsity

    rng = np.random.default_rng(n)
    D = sp.diags([rng.uniform(-1.0, -0.5, n - d) for d in band], list(band), shape=(n, n))
    M = (D + D.T).tocsr()
    M = (M + sp.diags(2.0 * np.asarray(abs(M).sum(axis=1)).ravel())).tocsr()
    M.sort_indices()
    want = rng.standard_normal(n)
    ctx = cx.get_cuda_context()
    A = CUDAMatrix(ctx, Sparsity.from_csr(ctx, M.indptr.astype(np.int32), M.indices.astype(np.int32), n))
    A.values.copy_(torch.from_numpy(M.data))
    v = CUDAVector(ctx, n)
    v.vector.copy_(torch.from_numpy(M @ want))
    x, its, res = cx.CUDAAssembler().solve(A, v, rtol=1e-13)
    assert res <= 1e-13
    assert np.linalg.norm(x.to_host() - want) <= 1e-11 * np.linalg.norm(want)
    again, its2, _ = cx.CUDAAssembler().solve(A, v, rtol=1e-13)
    assert its == its2 and np.array_equal(x.to_host(), again.to_host())
