"""The FP64 solver at the edges of its kernels: fewer rows than a tile, tiles
with a remainder, rows longer than a stream of products, and both sides of the
size rule; against scipy's direct solve.  CG stops at |r| <= rtol |b|, so the
error is below rtol * cond in the 2-norm: the matrices here have a condition
number below 1e3, and 1e-12 leaves 1e-9."""
import numpy as np
import pytest

from conftest import ensure_library

pytestmark = pytest.mark.gpu


def _solve(M, b, rtol=1e-12):
    import torch

    import cudolfinx as cx
    from cudolfinx.la import CUDAMatrix, CUDAVector, Sparsity

    ctx = cx.get_cuda_context()
    S = Sparsity.from_csr(ctx, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.shape[0])
    A = CUDAMatrix(ctx, S)
    A.values.copy_(torch.from_numpy(M.data))
    v = CUDAVector(ctx, len(b))
    v.vector.copy_(torch.from_numpy(b))
    return cx.CUDAAssembler().solve(A, v, rtol=rtol)


def _spd(n, band, seed):
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    off = [d for d in band if d < n]
    D = sp.csr_matrix((n, n)) if not off else sp.diags([rng.uniform(-1.0, 0.0, n - d) for d in off], off, shape=(n, n))
    M = (D + D.T).tocsr()
    M = (M + sp.diags(np.asarray(abs(M).sum(axis=1)).ravel() + 1.0)).tocsr()
    M.sort_indices()
    return M


@pytest.mark.parametrize("n,band", [(1, [1]), (5, [1]), (63, [1, 2]), (64, [1, 2, 3, 5, 7, 11]), (65, [1, 9]),
                                    (300, range(1, 40)), (2500, [1, 40, 41]), (2500, range(1, 2400)),
                                    (1000, range(1, 18)), (1023, range(1, 30, 2))])
def test_sizes(n, band):
    ensure_library()
    import scipy.sparse.linalg as sla

    M = _spd(n, list(band), seed=n)
    b = np.random.default_rng(n + 1).standard_normal(n)
    x, its, res = _solve(M, b)
    want = sla.spsolve(M.tocsc(), b)
    assert res <= 1e-12
    assert np.linalg.norm(x.to_host() - want) <= 1e-9 * np.linalg.norm(want)
    again, its2, res2 = _solve(M, b)
    assert its == its2 and res == res2 and np.array_equal(x.to_host(), again.to_host())


def test_stops_at_max_iter_and_without_a_right_hand_side():
    ensure_library()
    import cudolfinx as cx  # noqa: F401

    M = _spd(5000, [1, 70], seed=3)
    b = np.ones(5000)
    x, its, res = _solve(M, np.zeros(5000))
    assert its == 0 and not x.to_host().any()
    for most in (0, 1, 7, 8, 9):
        from cudolfinx.la import CUDAMatrix, CUDAVector, Sparsity
        import torch

        ctx = cx.get_cuda_context()
        S = Sparsity.from_csr(ctx, M.indptr.astype(np.int32), M.indices.astype(np.int32), 5000)
        A = CUDAMatrix(ctx, S)
        A.values.copy_(torch.from_numpy(M.data))
        v = CUDAVector(ctx, 5000)
        v.vector.copy_(torch.from_numpy(b))
        _, its, _ = cx.CUDAAssembler().solve(A, v, rtol=1e-14, max_iter=most, raise_on_failure=False)
        assert its == most
