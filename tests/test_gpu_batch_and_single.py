"""fcu_pcg between two batched solves on one matrix: the batch's plan, tuning and captured launches stay. Seen from the
number of kernels a repeated batch launches (planning adds some) and from fcu_batch_config; the results repeat bit for
bit."""
import numpy as np
import pytest

from test_gpu_batch_resident import _batch, _block

pytestmark = pytest.mark.gpu


def _config(fcu, M, prec):
    import ctypes as C
    v = [C.c_int(), C.c_int(), C.c_int()]
    assert fcu._L().fcu_batch_config(M.h, prec, *[C.byref(x) for x in v]) == 0
    return [x.value for x in v]


@pytest.mark.parametrize("sizes,pattern", [
    ([900, 4000, 300], (1, 2)),                # the whole matrix is solved on chip as well
    ([25000, 20000, 9000], (1, 8000)),         # tried there, but neither precision fits
    ([3000, 2500], tuple(range(1, 17))),       # rows that only the queue takes: its shape is timed
])
def test_single_solves_keep_the_batch(fcu, ctx, sizes, pattern):
    rng = np.random.default_rng(sizes[0])
    A, M, offs = _batch(fcu, ctx, [_block(n, pattern, rng) for n in sizes])
    b = rng.standard_normal(A.shape[0])
    for prec in (fcu.FCU_FP64, fcu.FCU_MIXED):
        batch = lambda: M.batch_pcg(offs, b, tol=1e-12, max_iter=2000, precision=prec)[0]
        single = lambda: M.pcg(b, tol=1e-12, max_iter=2000, precision=prec)[0]
        x, y = batch(), single()
        config = _config(fcu, M, prec)
        n0 = ctx.kernel_launches
        assert np.array_equal(batch(), x)
        n1 = ctx.kernel_launches
        assert np.array_equal(single(), y)
        n2 = ctx.kernel_launches
        assert np.array_equal(batch(), x)
        n3 = ctx.kernel_launches
        assert np.array_equal(single(), y)
        n4 = ctx.kernel_launches
        assert np.array_equal(batch(), x) and np.array_equal(batch(), x)
        repeated = (ctx.kernel_launches - n4) // 2
        assert n1 - n0 == n3 - n2 == repeated and n2 - n1 == n4 - n3
        assert _config(fcu, M, prec) == config
        assert np.linalg.norm(b - A @ y) < 3e-12 * np.linalg.norm(b)
    M.close()
