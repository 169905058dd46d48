"""A far-field level whose boundary strip has more cells than one grid holds
blocks of 256 along z (65535): one 2D patch one cell wide.  With a state that
does not vary along it, cells out of the ends' reach equal those of a short
patch bitwise, and so do the ends."""
import numpy as np
import pytest

import mfgpu

pytestmark = pytest.mark.gpu
STATE = [1.0, 0.3, 0.2, 0.1, 2.0, 0.1, 0.2, 0.3]
FAR = [0.6, 0.1, 0.4, 0.2, 0.7, 0.3, 0.1, 0.2]


def _step(prec, n):
    p = mfgpu.orszag_params(64, time_approximation=mfgpu.TA_FIRST_ORDER, precision=prec)
    p.bc_kind = mfgpu.BC_FARFIELD
    for d, hi in enumerate((n - 1, 0)):
        p.domain_hi[d], p.periodic[d] = hi, 0
    for q, v in enumerate(FAR):
        p.bc_plasma[q] = v
    ctx = mfgpu.Context(p)
    lev = mfgpu.Level(ctx, [([0, 0, 0], [n - 1, 0, 0])])
    U = np.repeat(np.array(STATE)[:, None], n, axis=1)
    lev.upload_valid(U.ctypes.data)
    st, ndt, _, _ = lev.step(1e-3)
    assert st == mfgpu.MF_OK
    lev.download_valid(U.ctypes.data)
    lev.close()
    ctx.close()
    return U, ndt


@pytest.mark.parametrize("prec", [mfgpu.PREC_FP64, mfgpu.PREC_MIXED])
def test_long_strip_equals_short(gpulib, prec):
    n = 8388500
    assert (2 * n + 255) // 256 > 65535
    long, dt_long = _step(prec, n)
    short, dt_short = _step(prec, 64)
    assert not np.array_equal(short[:, 32], STATE)
    assert np.array_equal(long[:, :32], short[:, :32])
    assert np.array_equal(long[:, -32:], short[:, -32:])
    for q in range(len(STATE)):
        assert np.all(long[q, 31:-31] == short[q, 32])
    assert dt_long == dt_short
