"""Boundary facets and dofs where the matching of facets can go wrong: one cell,
facets shared by three or more cells, cells listed twice (none of their facets
is single), cells with a repeated vertex, meshes of a few to several hundred
thousand facets. Reference: a facet is on the boundary when its sorted vertices
occur exactly once over all cells; integers, compared exactly."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _facets(cells):
    d = cells.shape[1] - 1
    if d == 2:
        loc = [(1, 2), (2, 0), (0, 1)]
    else:
        loc = [tuple(i for i in range(4) if i != l) for l in range(4)]
    return np.sort(cells[:, loc], axis=2)          # cells x facets x vertices


def _single(cells):
    f = _facets(cells)
    flat = f.reshape(-1, f.shape[2])
    _, inv, cnt = np.unique(flat, axis=0, return_inverse=True, return_counts=True)
    ids = np.nonzero(cnt[inv.ravel()] == 1)[0]
    order = np.lexsort(flat[ids].T[::-1])
    return flat[ids][order], ids[order]


def _meshes(fcu):
    rng = np.random.default_rng(3)
    tri = np.array([[0, 1, 2]])
    yield "one triangle", rng.random((3, 2)), tri
    yield "the same triangle twice, turned", rng.random((4, 2)), np.array([[0, 1, 2], [1, 2, 0], [1, 2, 3]])
    yield "edge shared by three", rng.random((5, 2)), np.array([[0, 1, 2], [0, 1, 3], [1, 0, 4]])
    yield "repeated vertex", rng.random((5, 2)), np.array([[0, 1, 1], [1, 2, 3], [3, 2, 4]])
    yield "one tet", rng.random((4, 3)), np.array([[3, 1, 0, 2]])
    yield "face shared by three", rng.random((6, 3)), np.array([[0, 1, 2, 3], [2, 1, 0, 4], [5, 0, 2, 1]])
    yield "random tets", rng.random((40, 3)), rng.integers(0, 40, size=(3000, 4))
    for m in (fcu.unit_square(1, 1), fcu.unit_square(37, 5), fcu.unit_square(300, 201), fcu.unit_cube(1, 2, 1),
              fcu.unit_cube(31, 9, 17)):
        yield "grid", m.coords, rng.permutation(m.cells)


def test_boundary_against_counts(fcu, ctx):
    for name, X, cells in _meshes(fcu):
        mesh = fcu.Mesh(np.ascontiguousarray(X), np.ascontiguousarray(cells, dtype=np.int64))
        fv, ids = _single(np.asarray(cells))
        bd = fcu.boundary_dofs_2d(mesh, ctx) if mesh.dim == 2 else fcu.boundary_dofs_3d(mesh, ctx)
        assert np.array_equal(bd, np.unique(fv)), name
        v, c, lo = fcu.extract_boundary_facets(mesh, ctx)
        assert np.array_equal(np.sort(v, axis=1), fv), name
        assert np.array_equal(np.asarray(c) * (mesh.dim + 1) + np.asarray(lo), ids), name
        if mesh.dim == 3:
            V = fcu.FunctionSpace(ctx, mesh, fcu.FCU_SPACE_P2)
            _, ev = V.p2_dofmap()
            edge = {tuple(e): mesh.nv + i for i, e in enumerate(np.sort(ev, axis=1).tolist())}
            want = set(np.unique(fv).tolist())
            for a, b, d in fv.tolist():
                want |= {edge[(a, b)], edge[(b, d)], edge[(a, d)]}
            assert np.array_equal(V.boundary_dofs(), sorted(want)), name
            V.close()
