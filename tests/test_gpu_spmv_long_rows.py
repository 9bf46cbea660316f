"""SpMV of scalar matrices of 8 to 64 entries per row with one much longer row: its length decides which kernel runs.

The results are sums of at most n products: within 4 eps log2(n) sum |a_ij x_j| of the reference. The time is compared
with that of the same matrix without the long row. A row of 20,000 entries spread over a CTA takes about 20 us beside
the 5 us of the rest; walked by the four lanes of a short row it takes some 600 trips, 400 us or more.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _stencil(n, dim):
    T = sp.diags([np.ones(n - 1), np.ones(n), np.ones(n - 1)], [-1, 0, 1])
    A = T
    for _ in range(dim - 1):
        A = sp.kron(A, T)
    return A.tocsr()


def _with_row(A, length, rng):
    n = A.shape[0]
    if not length:
        return A
    c = rng.choice(n, size=length, replace=False)
    return (A + sp.coo_matrix((rng.standard_normal(length), (np.full(length, n // 2), c)), shape=(n, n))).tocsr()


def _wrap(fcu, ctx, A):
    A = sp.csc_matrix(A)
    A.sort_indices()
    return fcu.Matrix.from_csc(ctx, fcu.CscMatrix(A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64),
                                                  A.data.astype(np.float64)))


# around the limits of both lane counts (64 and 128 entries for small matrices), the stream kernel's block, the largest
@pytest.mark.parametrize("n,dim", [(20, 2), (60, 2), (12, 3), (25, 3)])
@pytest.mark.parametrize("length", [40, 64, 65, 128, 129, 2030, 2100, 15000])
def test_long_row_results(fcu, ctx, n, dim, length):
    rng = np.random.default_rng(length)
    A = _with_row(_stencil(n, dim), min(length, n**dim), rng)
    x = rng.standard_normal(A.shape[0])
    M = _wrap(fcu, ctx, A)
    copy = M.clone()
    bound = 4 * np.finfo(float).eps * np.log2(A.shape[0]) * np.asarray(abs(A) @ np.abs(x)).ravel()
    for m in (M, copy):
        assert np.all(np.abs(m.spmv(x) - A @ x) <= bound)
        m.close()


def _time(M, ctx, n):
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = np.inf
    for _ in range(6):
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
            e[0].record()
            for _ in range(10):
                M.spmv(x, y)
            e[1].record()
        e[1].synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best


def test_long_row_time(fcu, ctx):
    rng = np.random.default_rng(0)
    A = _stencil(40, 3)
    t = []
    for length in (0, 20000):
        M = _wrap(fcu, ctx, _with_row(A, length, rng))
        t.append(_time(M, ctx, A.shape[0]))
        M.close()
    assert t[1] < 20 * t[0], t
