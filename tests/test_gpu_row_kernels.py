"""Row kernels at the sizes where their split can go wrong.

P2 stiffness (three rows a warp, contributions in chunks of ten): meshes of one
cell, row counts of every remainder by three, vertices with more than ten and
more than thirty cells, degenerate cells. Entries are sums of at most some
hundred products of a few roundings each, relative to the largest entry:
tolerance 1e-13 of it.

Dirichlet elimination from the listed rows: non-symmetric patterns, empty lists,
every dof eliminated, repeated dofs. The matrix entries are copied or set, so
they agree exactly; the right-hand side sums at most one product per entry of a
row: 1e-13 of sum |a_ij g_j| + |b_i|.

SpMV of rows of 8 to 64 entries: ragged rows, empty rows, row counts around a
warp's. Each result is a sum of at most n products: within
4 eps sum |a_ij x_j| for the lengths used (about 2 log2 of the tree depth plus the
lane sums of at most eight terms and their order in the reference).
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O

pytestmark = pytest.mark.gpu


def _wrap(fcu, ctx, A):
    A = sp.csc_matrix(A)
    A.sort_indices()
    return fcu.Matrix.from_csc(ctx, fcu.CscMatrix(A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64),
                                                  A.data.astype(np.float64)))


def _meshes():
    rng = np.random.default_rng(0)
    X = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    yield X, np.array([[0, 1, 2, 3]])
    yield X, np.array([[3, 1, 0, 2]])
    # fan: 40 cells around the edge (0, 1); vertices 0 and 1 have 40 cells each
    th = 2 * np.pi * np.arange(40) / 40
    fan = np.concatenate([[[0, 0, 0], [0, 0, 1.0]], np.stack([np.cos(th), np.sin(th), 0.5 + 0 * th], 1)])
    yield fan, np.array([[0, 1, 2 + i, 2 + (i + 1) % 40] for i in range(40)])
    for n in ((1, 1, 1), (2, 1, 1), (3, 2, 2), (5, 4, 3)):
        m = O.unit_cube(*n)
        yield m.coords + rng.uniform(-0.05, 0.05, m.coords.shape), m.cells
    m = O.unit_cube(2, 2, 2)  # a flat cell among the others
    flat = np.concatenate([m.cells, [[m.cells[0][0], m.cells[0][1], m.cells[0][2], m.cells[0][2]]]])
    yield m.coords, flat


def test_p2_stiffness_rows(fcu, ctx):
    rng = np.random.default_rng(1)
    for X, cells in _meshes():
        om = O.Mesh(np.ascontiguousarray(X), np.ascontiguousarray(cells, dtype=np.int64))
        kappa = np.exp(rng.standard_normal(len(cells)))
        cd, nd = O.p2_dofmap(om)[0], None
        V = fcu.FunctionSpace(ctx, fcu.Mesh(om.coords, om.cells), fcu.FCU_SPACE_P2)
        nd = V.ndofs
        for kap in (kappa, None):
            M = fcu.Matrix(ctx, V).assemble_stiffness(kap)
            A = M.export_csc().to_scipy().toarray()
            B = O.assemble_p2_stiffness_3d(om, cd, nd, kap).to_scipy().toarray()
            assert np.max(np.abs(A - B)) <= 1e-13 * np.max(np.abs(B)), (len(cells), np.max(np.abs(A - B)))
            M.close()
        V.close()


def test_p2_node_that_is_a_corner_of_one_cell_and_a_midpoint_of_another(fcu, ctx):
    """Callers number the nodes of P2_NODES spaces themselves: a row may mix
    contributions of a corner and of a mid-edge node, here with more than ten of
    the corner's."""
    rng = np.random.default_rng(4)
    m = O.unit_cube(2, 2, 2)
    cd, _ = O.p2_dofmap(m)
    nd = int(cd.max()) + 1
    X = np.concatenate([m.coords, rng.random((nd - m.nv, 3))])
    cells = np.asarray(m.cells, dtype=np.int64)
    centre = int(np.argmax(np.bincount(cells.ravel())))
    cd = np.array(cd)
    away = [c for c in range(len(cells)) if centre not in cells[c]]
    for c in away[:2]:
        cd[c, 7] = centre
    kappa = np.exp(rng.standard_normal(len(cells)))
    mesh = fcu.Mesh(np.ascontiguousarray(X), cells)
    V = fcu.FunctionSpace(ctx, mesh, fcu._abi.FCU_SPACE_P2_NODES, np.ascontiguousarray(cd, dtype=np.int64))
    M = fcu.Matrix(ctx, V).assemble_stiffness(kappa)
    A = M.export_csc().to_scipy().toarray()
    B = O.assemble_p2_stiffness_3d(O.Mesh(X, cells), cd, nd, kappa).to_scipy().toarray()
    assert A.shape == B.shape
    assert np.max(np.abs(A - B)) <= 1e-13 * np.max(np.abs(B))
    M.close()
    V.close()


def _ragged(n, mean, rng, symmetric):
    rows, cols = [], []
    for i in range(n):
        k = int(rng.integers(0, 2 * mean + 1))
        c = np.unique(np.clip(i + rng.integers(-3 * mean, 3 * mean + 1, size=k), 0, n - 1))
        rows.append(np.full(len(c), i))
        cols.append(c)
    r, c = np.concatenate(rows), np.concatenate(cols)
    A = sp.csr_matrix((rng.standard_normal(len(r)), (r, c)), shape=(n, n))
    if symmetric:
        A = A + A.T
    return (A + sp.diags(np.full(n, 3.0))).tocsc()


@pytest.mark.parametrize("n,symmetric", [(1, True), (31, True), (300, True), (300, False), (2500, False)])
@pytest.mark.parametrize("share", [0.0, 0.03, 1.0])
def test_dirichlet_rows(fcu, ctx, n, symmetric, share):
    rng = np.random.default_rng(n)
    A = _ragged(n, 6, rng, symmetric)
    dofs = np.sort(rng.choice(n, size=int(np.ceil(share * n)), replace=False)).astype(np.int64)
    vals = rng.standard_normal(len(dofs))
    b = rng.standard_normal(n)
    if len(dofs) > 3:  # repeated, with their values
        dofs, vals = np.concatenate([dofs, dofs[:3]]), np.concatenate([vals, vals[:3]])
    M = _wrap(fcu, ctx, A)
    bb = b.copy()
    M.apply_dirichlet(bb, dofs, vals)
    C = M.export_csc().to_scipy().toarray()
    As = sp.csc_matrix(A)
    As.sort_indices()
    R, rb = O.apply_dirichlet_bc(O.Csc(n, As.indptr.astype(np.int64), As.indices.astype(np.int64), As.data), b, dofs,
                                 vals)
    assert np.array_equal(C, R.to_scipy().toarray())
    g = np.zeros(n)
    g[dofs] = vals
    bound = 1e-13 * (abs(As) @ np.abs(g) + np.abs(b) + np.abs(g))
    assert np.all(np.abs(bb - rb) <= bound)
    M.close()


@pytest.mark.parametrize("n", [1, 7, 33, 1023, 4099])
@pytest.mark.parametrize("mean", [9, 15, 27, 40, 62])
def test_spmv_medium_rows(fcu, ctx, n, mean):
    rng = np.random.default_rng(n * 100 + mean)
    A = _ragged(n, mean, rng, False)
    x = rng.standard_normal(n)
    M = _wrap(fcu, ctx, A)
    y = M.spmv(x)
    bound = 4 * np.finfo(float).eps * np.asarray(abs(A) @ np.abs(x)).ravel() * max(1.0, np.log2(mean))
    assert np.all(np.abs(y - A @ x) <= bound)
    M.close()
