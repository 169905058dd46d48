"""The autotuner picks block sizes by timing only where a launch of the level
depends on them: kernels with fixed blocks (the FP64 face fluxes split by
fluid, the update by fluid) keep the default, so two tuned levels of one kind
launch alike."""
import numpy as np
import pytest

import mfgpu

pytestmark = pytest.mark.gpu
DEFAULT = 128


def _tuned(p, n, patch, sd, init, times):
    ctx = mfgpu.Context(p)
    lev = mfgpu.Level(ctx, mfgpu.tile_boxes(n, patch, sd))
    buf = np.zeros(lev.ndoubles)
    for i in range(len(lev.boxes)):
        lev.patch_view(buf, i)[:] = mfgpu.init_host_fab(p, *lev.fab_box(i), init)
    lev.upload(buf.ctypes.data)
    out = [lev.autotune(2) for _ in range(times)]
    lev.close()
    ctx.close()
    return out


@pytest.mark.parametrize("prec", [mfgpu.PREC_FP64, mfgpu.PREC_FP64_FAST])
@pytest.mark.parametrize("problem", ["orszag", "helio", "hancock"])
def test_fixed_blocks_are_not_tuned(gpulib, prec, problem):
    if problem == "orszag":
        args = (mfgpu.orszag_params(64, precision=prec), 64, 16, 2, "orszag")
    else:
        ta = mfgpu.TA_HANCOCK if problem == "hancock" else mfgpu.TA_RK2
        args = (mfgpu.helio_params(32, time_approximation=ta, precision=prec), 32, 16, 3, "helio")
    for _, flux, update in _tuned(*args, times=6):
        assert (flux, update) == (DEFAULT, DEFAULT)


def test_tuned_blocks_stay_candidates(gpulib):
    """Kernels whose blocks follow the batch are still tuned."""
    p = mfgpu.helio_params(32, region_tracer=True)
    for shapes in _tuned(p, 32, 16, 3, "helio", times=2):
        assert all(s in (64, 128, 256) for s in shapes)
    p = mfgpu.helio_params(32, precision=mfgpu.PREC_MIXED)
    for shapes in _tuned(p, 32, 16, 3, "helio", times=2):
        assert all(s in (64, 128, 256) for s in shapes)
