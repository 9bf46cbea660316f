"""The batched PCG's on-chip form at the sizes where its split can go wrong:
empty and one-row instances, shares around the thread count and around the rows
a CTA keeps, instances of every cluster size, more instances of one size than
clusters run at a time, rows left in global memory (the largest FP64 instances)
and instances that only the streaming form takes (too many rows, long rows).

Every block is symmetric and its diagonal exceeds the sum of the row's other
entries by 5 % or more, so cond(A) <= 41 and CG needs under 100 iterations for
1e-12; the recurrence's residual then drifts from b - A x by some 100 eps
|A||x| <= 1e-12 |b|: the true residual stays below 3e-12.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _block(n, offs, rng):
    A = sp.csr_matrix((n, n))
    for o in offs:
        if 0 < o < n:
            d = -rng.uniform(0.1, 1.0, n - o)
            A = A + sp.diags([d, d], [o, -o], shape=(n, n), format="csr")
    return (A + sp.diags(1.05 * np.asarray(abs(A).sum(axis=1)).ravel() + 0.1, format="csr")).tocsr()


def _batch(fcu, ctx, blocks):
    A = sp.csc_matrix(sp.block_diag([B for B in blocks if B.shape[0]], format="csc"))
    A.sort_indices()
    M = fcu.Matrix.from_csc(ctx, fcu.CscMatrix(A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64),
                                               A.data.astype(np.float64)))
    return A, M, np.concatenate([[0], np.cumsum([B.shape[0] for B in blocks])])


GRID = lambda n: (1, int(np.sqrt(n)) or 1, int(np.sqrt(n)) + 1)  # rows of a triangle grid


@pytest.mark.parametrize("sizes,pattern", [
    ([1, 2, 0, 511, 512, 513, 1025], GRID),
    ([4607, 4608, 4609, 9217, 0, 17, 20000, 33000], GRID),
    ([60000] * 9 + [40000, 5000, 300], GRID),
    ([16 * 4608, 16 * 4608 + 1, 700], lambda n: (1, 2)),
    ([1], GRID),
    ([20001], GRID),
    ([3000, 64, 900], lambda n: tuple(range(1, 16))),   # 31 entries to a row
    ([3000, 64, 900], lambda n: tuple(range(1, 17))),   # 33: streaming form
    ([5000, 4000], lambda n: (1, n // 2, n - 1)),       # as wide as the instance
])
def test_resident_batch_residuals(fcu, ctx, sizes, pattern):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    blocks = [_block(n, pattern(n), rng) for n in sizes]
    A, M, offs = _batch(fcu, ctx, blocks)
    b = rng.standard_normal(A.shape[0])
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED):
        first = None
        for _ in range(2):
            x, it, rel, st, _ = M.batch_pcg(offs, b, tol=1e-12, max_iter=2000, precision=prec)
            assert np.all(st == 0)
            for i, B in enumerate(blocks):
                sl = slice(offs[i], offs[i + 1])
                if B.shape[0]:
                    r = np.linalg.norm(b[sl] - B @ x[sl]) / np.linalg.norm(b[sl])
                    assert r < 3e-12, (prec, i, r)
                    assert rel[i] < 1e-12
                else:
                    assert it[i] == 0
            assert first is None or np.array_equal(first, x)
            first = x
    M.close()


def test_offsets_refused_twice_then_accepted(fcu, ctx):
    rng = np.random.default_rng(0)
    blocks = [_block(n, (1, 5), rng) for n in (40, 60)]
    A, M, offs = _batch(fcu, ctx, blocks)
    b = rng.standard_normal(100)
    for _ in range(2):
        with pytest.raises(fcu.FcuError, match="block diagonal"):
            M.batch_pcg([0, 41, 100], b)
    x, _, _, st, _ = M.batch_pcg(offs, b, tol=1e-12)
    assert np.all(st == 0) and np.linalg.norm(b - A @ x) < 3e-12 * np.linalg.norm(b)
    M.close()


@pytest.mark.parametrize("n,pattern", [
    (60000, lambda n: (1, 250)),                 # the largest that is tried on chip
    (60001, lambda n: (1, 250)),
    (30000, lambda n: tuple(range(1, 8))),       # FP64 does not fit, FP32 does
    (30000, lambda n: (1, 14999)),               # fits but for its bandwidth
    (5000, lambda n: tuple(range(1, 17))),       # rows too long
])
def test_single_systems_on_both_sides_of_the_on_chip_limit(fcu, ctx, n, pattern):
    rng = np.random.default_rng(n)
    A, M, _ = _batch(fcu, ctx, [_block(n, pattern(n), rng)])
    b = rng.standard_normal(n)
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED, fcu.FCU_FP64):
        x, info = M.pcg(b, tol=1e-12, max_iter=2000, precision=prec)
        assert info.status == 0 and np.linalg.norm(b - A @ x) < 3e-12 * np.linalg.norm(b)
    # a solve of one system between two batches on the same matrix
    y, _, _, st, _ = M.batch_pcg([0, n], b, tol=1e-12, max_iter=2000)
    assert np.all(st == 0) and np.linalg.norm(b - A @ y) < 3e-12 * np.linalg.norm(b)
    M.close()
