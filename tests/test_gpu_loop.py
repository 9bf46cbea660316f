"""The persistent PCG loop on the matrices where its tiling can go wrong.

Each system is solved through the C ABI in FP64 and in mixed precision and
compared with scipy's direct solve of the exported matrix: sizes around the
tile and CTA counts, odd orders (the vectors are updated in pairs of
elements), rows of very different lengths (tiles cut by entries), a matrix
with an empty-but-diagonal row pattern, 3x3 blocks with one long row, and
sizes on both sides of the switch between the two forms of the loop.
Tolerance: a solve stopped at relative residual 1e-12 has a relative error of
at most cond(A) * 1e-12; the systems are shifted so that cond(A) <= 1e4, so
1e-8 holds with room for the direct solve's own rounding.
"""
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _wrap(fcu, ctx, A):
    A = sp.csc_matrix(A)
    A.sort_indices()
    return fcu.Matrix.from_csc(ctx, fcu.CscMatrix(A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64),
                                                  A.data.astype(np.float64)))


def _banded(n, half, rng):
    """Symmetric, diagonally dominant, about 2 * half + 1 entries per row."""
    offs = np.unique(rng.integers(1, max(2, min(n, 40 * half)), size=half)) if n > 1 else np.empty(0, int)
    A = sp.lil_matrix((n, n)).tocsr()
    for o in offs:
        if o < n:
            d = -rng.uniform(0.1, 1.0, n - o)
            A = A + sp.diags([d, d], [o, -o], shape=(n, n))
    return (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1e-2)).tocsc()


# scalar systems solved from x0 (the small-system path starts from zero only), so every size takes the loop
@pytest.mark.parametrize("n,half", [(1, 1), (3, 1), (147, 2), (149, 3), (480 * 148 + 1, 3), (40001, 7), (30011, 20),
                                    (200003, 5), (500001, 4), (3001, 60)])
def test_scalar_systems_match_direct_solve(fcu, ctx, n, half):
    rng = np.random.default_rng(n)
    A = _banded(n, half, rng)
    M = _wrap(fcu, ctx, A)
    b = rng.standard_normal(n)
    x0 = 1e-3 * rng.standard_normal(n)
    ref = spl.spsolve(A, b) if n <= 50000 else None
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED):
        x, info = M.pcg(b, x0=x0, tol=1e-12, max_iter=5000, precision=prec)
        assert info.status == 0
        r = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        assert r < 2e-12, (prec, r)
        if ref is not None:
            assert np.linalg.norm(x - ref) <= 1e-8 * np.linalg.norm(ref)
        again, info2 = M.pcg(b, x0=x0, tol=1e-12, max_iter=5000, precision=prec)
        assert info2.iterations == info.iterations and np.array_equal(x, again)
    M.close()


@pytest.mark.parametrize("long_row", [2001, 5001])
def test_ragged_rows(fcu, ctx, long_row):
    """One row and column coupled to many others beside short rows: tiles cut by entries, or (a row longer than a
    tile) the per-iteration kernels."""
    n = 5001
    rng = np.random.default_rng(5)
    A = _banded(n, 2, rng).tolil()
    A[0, :long_row] = -1e-3
    A[:long_row, 0] = -1e-3
    A[0, 0] = 10.0
    A = (A.tocsr() + sp.diags(np.full(n, 1e-2))).tocsc()
    M = _wrap(fcu, ctx, A)
    b = rng.standard_normal(n)
    ref = spl.spsolve(A, b)
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED):
        x, info = M.pcg(b, x0=np.zeros(n), tol=1e-12, max_iter=5000, precision=prec)
        assert info.status == 0 and np.linalg.norm(x - ref) <= 1e-8 * np.linalg.norm(ref)
    M.close()


# 3x3 blocks: fewer rows than CTAs, one tile, an odd order, both sides of the pairs' limit (FP64 and FP32 differ)
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 4, 3), (30, 9, 7), (44, 20, 20), (60, 22, 21), (70, 30, 30)])
def test_block_systems_match_the_graph_kernels(fcu, ctx, dims):
    m = fcu.box_beam(1.0, 1.0, 1.0, *dims)
    V = fcu.FunctionSpace(ctx, m, fcu.FCU_SPACE_P1_VEC3)
    K = fcu.Matrix(ctx, V).assemble_elasticity(1.0, 0.3)
    Mm = fcu.Matrix(ctx, V).assemble_mass(50.0)
    K.set_add_scaled(K, Mm, 1.0)
    rng = np.random.default_rng(7)
    b = rng.standard_normal(V.ndofs)
    xs = {}
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED):
        x, info = K.pcg(b, tol=1e-12, max_iter=5000, precision=prec)
        assert info.status == 0
        y = K.spmv(x)
        assert np.linalg.norm(b - y) <= 2e-12 * np.linalg.norm(b)
        xs[prec] = x
    assert np.linalg.norm(xs[fcu.FCU_FP64] - xs[fcu.FCU_MIXED]) <= 1e-8 * np.linalg.norm(xs[fcu.FCU_FP64])
    # limits: exactly the asked iterations, the iterate kept, restart continues
    x3, info3 = K.pcg(b, tol=1e-14, max_iter=3, raise_on_error=False)
    assert info3.iterations == 3 and info3.status == 3
    xc, infoc = K.pcg(b, x0=x3, tol=1e-12, max_iter=5000)
    assert infoc.status == 0 and np.linalg.norm(xc - xs[fcu.FCU_FP64]) <= 1e-8 * np.linalg.norm(xc)
    for h in (K, Mm, V):
        h.close()


def test_block_csr_caller_matrix_with_a_long_row(fcu, ctx):
    """A caller's 3x3-block matrix whose first row couples to 90 others: tiles of few rows."""
    n = 400
    rng = np.random.default_rng(11)
    P = _banded(n, 3, rng).tolil()
    P[0, 1:91] = -0.01
    P[1:91, 0] = -0.01
    P = P.tocsr()
    P.sort_indices()
    nnz = P.nnz
    blocks = np.empty((nnz, 3, 3))
    S = rng.uniform(-0.02, 0.02, (3, 3))
    S = S + S.T
    for k, v in enumerate(P.data):
        blocks[k] = v * (np.eye(3) + S)
    A = sp.bsr_matrix((blocks, P.indices, P.indptr), shape=(3 * n, 3 * n)).tocsc()
    A = (A + 2.0 * sp.identity(3 * n)).tocsc()
    Ab = sp.bsr_matrix(A, blocksize=(3, 3))
    Ab.sort_indices()
    M = fcu.Matrix.from_bsr3(ctx, n, Ab.indptr, Ab.indices, Ab.data.reshape(-1))
    b = rng.standard_normal(3 * n)
    ref = spl.spsolve(A, b)
    x, info = M.pcg(b, tol=1e-12, max_iter=5000)
    assert info.status == 0 and np.linalg.norm(x - ref) <= 1e-8 * np.linalg.norm(ref)
    M.close()


def test_p2_and_p1_spaces_match_the_graph(fcu, ctx, tmp_path):
    """P2 (tiles cut by entries) and P1 in 3D (equal tiles) against the per-iteration kernels in a child process."""
    child = (
        "import sys, numpy as np\n"
        f"sys.path.insert(0, {ROOT + '/fenics-rs_b200'!r})\n"
        "import fenics_cuda as fcu\n"
        "ctx = fcu.Context(0); out = {}\n"
        "for name, kind, n in (('p2', fcu.FCU_SPACE_P2, 18), ('p1', fcu.FCU_SPACE_P1, 37)):\n"
        "    m = fcu.unit_cube(n, n - 1, n - 2); V = fcu.FunctionSpace(ctx, m, kind)\n"
        "    k = np.exp(np.random.default_rng(3).standard_normal(m.nc))\n"
        "    A = fcu.Matrix(ctx, V).assemble_stiffness(k); b = V.rhs_source(fcu.FCU_SRC_CONSTANT, params=(1.0,))\n"
        "    bd = V.boundary_dofs(); A.apply_dirichlet(b, bd, np.zeros(len(bd)))\n"
        "    for p in (fcu.FCU_FP64, fcu.FCU_MIXED):\n"
        "        x, i = A.pcg(b, tol=1e-11, max_iter=20000, precision=p); out[f'{name}{p}'] = x; out[f'{name}{p}it'] = i.iterations\n"
        "np.savez(sys.argv[1], **out)\n")
    res = {}
    for mode in ("0", "1"):
        f = str(tmp_path / f"m{mode}.npz")
        r = subprocess.run([sys.executable, "-c", child, f], env=dict(os.environ, FCU_PERSISTENT=mode),
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        res[mode] = np.load(f)
    for name in ("p2", "p1"):
        for p in (fcu.FCU_FP64, fcu.FCU_MIXED):
            x0, x1 = res["0"][f"{name}{p}"], res["1"][f"{name}{p}"]
            # both stop at 1e-11 on a system with condition number below 1e5
            assert np.linalg.norm(x0 - x1) <= 1e-6 * np.linalg.norm(x0)
            i0, i1 = int(res["0"][f"{name}{p}it"]), int(res["1"][f"{name}{p}it"])
            assert abs(i0 - i1) <= max(3, (0.02 if p == fcu.FCU_FP64 else 0.15) * i0)
