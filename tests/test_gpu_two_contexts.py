"""One mesh used from two contexts (each with its own stream). The mesh is complete when its creation returns, so work
on the second context neither waits for the first one's stream nor launches anything on it; results are equal bit for
bit to those on the mesh's own context."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _space(fcu, ctx, h, kind):
    out = C.c_void_p()
    assert fcu._L().fcu_space_create(ctx.h, h, kind, C.byref(out)) == 0
    return out


def _loads(fcu, ctx, h, nv):
    L, got = fcu._L(), {}
    for kind, n in ((fcu.FCU_SPACE_P1, nv), (fcu.FCU_SPACE_P1_VEC3, 3 * nv)):
        V = _space(fcu, ctx, h, kind)
        b = np.full(n, np.nan)
        if kind == fcu.FCU_SPACE_P1:
            for src, par in ((fcu.FCU_SRC_CONSTANT, [2.5, 0.0]), (fcu.FCU_SRC_SIN_PRODUCT, [1.5, 3.0])):
                p = np.array(par)
                assert L.fcu_assemble_rhs_source(ctx.h, V, src, p.ctypes.data, None, b.ctypes.data) == 0
                got[kind, src] = b.copy()
        else:
            f = np.array([0.5, -1.0, 2.0])
            assert L.fcu_assemble_body_force(ctx.h, V, f.ctypes.data, b.ctypes.data) == 0
            got[kind] = b.copy()
        L.fcu_space_destroy(V)
    return got


def test_load_vectors_on_another_contexts_mesh(fcu):
    m = fcu.box_beam(3.0, 1.0, 1.0, 17, 9, 11)
    with fcu.Context(0) as a, fcu.Context(0) as b:
        h = m.handle(a)
        launched = a.kernel_launches
        with torch.cuda.stream(torch.cuda.ExternalStream(a.stream)):
            torch.cuda._sleep(200_000_000)  # the mesh's own stream is busy for about 0.1 s
        other = _loads(fcu, b, h, m.nv)
        assert a.kernel_launches == launched
        own = _loads(fcu, a, h, m.nv)
        for k in own:
            assert np.isfinite(own[k]).all() and np.array_equal(own[k], other[k]), k
        m.release()


def _boundary(fcu, ctx, h, nv):
    L, n = fcu._L(), C.c_int64(nv)
    dofs = np.empty(nv, np.int64)
    assert L.fcu_boundary_dofs(ctx.h, h, dofs.ctypes.data, C.byref(n)) == 0
    out = [dofs[:n.value]]
    V = _space(fcu, ctx, h, fcu.FCU_SPACE_P2)
    assert L.fcu_space_boundary_dofs(ctx.h, V, None, C.byref(n)) == 0
    p2 = np.empty(n.value, np.int64)
    assert L.fcu_space_boundary_dofs(ctx.h, V, p2.ctypes.data, C.byref(n)) == 0
    L.fcu_space_destroy(V)
    assert L.fcu_boundary_facets(ctx.h, h, None, None, None, C.byref(n)) == 0
    fv, fc, fl = np.empty((n.value, 3), np.int64), np.empty(n.value, np.int64), np.empty(n.value, np.int64)
    assert L.fcu_boundary_facets(ctx.h, h, fv.ctypes.data, fc.ctypes.data, fl.ctypes.data, C.byref(n)) == 0
    return out + [p2, fv, fc, fl]


def test_boundary_of_another_contexts_mesh(fcu):
    m = fcu.box_beam(3.0, 1.0, 1.0, 17, 9, 11)
    with fcu.Context(0) as a, fcu.Context(0) as b:
        h = m.handle(a)
        launched = a.kernel_launches
        with torch.cuda.stream(torch.cuda.ExternalStream(a.stream)):
            torch.cuda._sleep(200_000_000)
        other = _boundary(fcu, b, h, m.nv)
        assert a.kernel_launches == launched
        for x, y in zip(_boundary(fcu, a, h, m.nv), other):
            assert np.array_equal(x, y)
        m.release()
