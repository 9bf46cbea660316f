"""Host threads with a context each, solving matrices of different sizes at the same time: the launches of one must
not change what another's are allowed. Every solve is stopped after three iterations, so that launches follow one
another quickly; three threads solve small systems for as long as the fourth solves large ones. Each result has to
equal, bit for bit, the one the same context gave alone (the loop adds in a fixed order)."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SOLVES = 2000


def _system(fcu, ctx, dims):
    V = fcu.FunctionSpace(ctx, fcu.box_beam(4.0, 1.0, 1.0, *dims), fcu.FCU_SPACE_P1_VEC3)
    M = fcu.Matrix(ctx, V).assemble_elasticity(1.0, 0.3)
    b = V.body_force([0.1, 0.0, -1.0])
    d = np.arange(3 * (dims[0] + 1), dtype=np.int64)
    M.apply_dirichlet(b, d, np.zeros(len(d)))
    return V, M, b


# the loop's shared memory differs several times over between the two meshes, in each precision
@pytest.mark.parametrize("prec", ["FCU_FP64", "FCU_MIXED"])
def test_loop_from_several_threads(fcu, prec):
    prec = getattr(fcu, prec)
    errors, over = [], threading.Event()
    start = threading.Barrier(4)

    def worker(dims, last):
        try:
            with fcu.Context(0) as ctx:
                V, M, b = _system(fcu, ctx, dims)
                bd, xd = torch.as_tensor(b, device="cuda"), torch.empty(V.ndofs, dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()

                def solve():
                    info = M.pcg(bd, x=xd, tol=1e-14, max_iter=3, precision=prec, raise_on_error=False)[1]
                    if info.status != 3:
                        raise AssertionError((dims, info.status, fcu._L().fcu_last_error(ctx.h)))

                solve()
                ref = xd.clone()
                start.wait(timeout=60)
                for k in range(SOLVES if last else 100 * SOLVES):
                    solve()
                    if k % 100 == 0 and not torch.equal(xd, ref):
                        raise AssertionError((dims, "another result"))
                    if over.is_set():
                        break
                M.close()
                V.close()
        except BaseException as e:
            errors.append(e)
            start.abort()
        finally:
            if last:
                over.set()

    threads = [threading.Thread(target=worker, args=a)
               for a in [((3, 2, 2), False)] * 3 + [((44, 20, 18), True)]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
