"""3x3-block rows too long for the tiled SpMV: block-Jacobi solves, which need it, are refused, and the refusal leaves
nothing behind - the point-Jacobi solve of the same matrix on the same context follows and is right."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def test_refused_solve_leaves_the_context_usable(fcu, ctx):
    n, long_row = 600, 200
    rng = np.random.default_rng(2)
    P = sp.diags([-np.ones(n - 1), -np.ones(n - 1)], [-1, 1]).tolil()
    P[0, 1:long_row] = -0.01
    P[1:long_row, 0] = -0.01
    P = P.tocsr()
    P = (P + sp.diags(np.asarray(abs(P).sum(axis=1)).ravel() + 0.5)).tocsr()
    P.sort_indices()
    blocks = P.data[:, None, None] * np.eye(3)
    A = sp.bsr_matrix((blocks, P.indices, P.indptr), shape=(3 * n, 3 * n)).tocsr()
    M = fcu.Matrix.from_bsr3(ctx, n, P.indptr, P.indices, blocks.reshape(-1))
    b = rng.standard_normal(3 * n)
    M.block_jacobi(True)
    for _ in range(2):
        with pytest.raises(fcu.FcuError):
            M.pcg(b, tol=1e-10, max_iter=500)
        M.block_jacobi(False)
        x, info = M.pcg(b, tol=1e-12, max_iter=500)
        # diagonally dominant by 0.5 of at most 5.5: well conditioned, the recurrence's residual drifts by rounding only
        assert info.status == 0 and np.linalg.norm(b - A @ x) < 3e-12 * np.linalg.norm(b)
        M.block_jacobi(True)
    M.close()
