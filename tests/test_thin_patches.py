"""Levels whose outermost patches are one or two cells wide: the far-field
ghosts of the patches next to them lie beyond a sibling's cells, so the
neutral populations copied into them come from a ghost cell that the sibling
copy has filled.  The step equals that of one patch that holds the whole
domain bitwise, in every precision."""
import numpy as np
import pytest

import mfgpu
from helpers import valid_view

pytestmark = pytest.mark.gpu
PREC = {"fp64": mfgpu.PREC_FP64, "fast": mfgpu.PREC_FP64_FAST, "mixed": mfgpu.PREC_MIXED,
        "ce32": mfgpu.PREC_MIXED_CE32}


def _cut(cuts):
    e = np.concatenate([[0], np.cumsum(cuts)]).tolist()
    r = range(len(cuts))
    return [([e[i], e[j], e[k]], [e[i + 1] - 1, e[j + 1] - 1, e[k + 1] - 1])
            for k in r for j in r for i in r]


@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("ta", [mfgpu.TA_FIRST_ORDER, mfgpu.TA_RK2])
@pytest.mark.parametrize("nf,cuts", [(4, (1, 10, 1)), (5, (2, 8, 2)), (3, (1, 1, 8))])
def test_thin_boundary_patches_equal_one_patch(gpulib, prec, ta, nf, cuts):
    n = sum(cuts)
    p = mfgpu.helio_params(n, time_approximation=ta, precision=PREC[prec])
    ng = mfgpu.num_ghost(p)
    U = mfgpu.init_host_fab(p, [-ng] * 3, [n - 1 + ng] * 3, "helio")
    U = U * (1.0 + 0.02 * np.random.default_rng(5).standard_normal(U.shape))
    U = np.concatenate([U[:9]] + [U[9 + 5 * (f % 3) : 14 + 5 * (f % 3)] for f in range(nf - 1)])
    p.n_fluids = nf
    outs = []
    for boxes in ([([0] * 3, [n - 1] * 3)], _cut(cuts)):
        ctx = mfgpu.Context(p)
        lev = mfgpu.Level(ctx, boxes)
        flat = np.zeros(lev.ndoubles)
        for i in range(len(boxes)):
            lo, hi = lev.fab_box(i)
            lev.patch_view(flat, i)[:] = U[(slice(None),) + tuple(
                slice(lo[d] + ng, hi[d] + ng + 1) for d in (2, 1, 0))]
        lev.upload(flat.ctypes.data)
        dt = 0.2 * lev.compute_dt()[0]
        new = [lev.step(dt)[1] for _ in range(2)]
        lev.download(flat.ctypes.data)
        whole = np.zeros((U.shape[0], n, n, n))
        for i, (blo, bhi) in enumerate(boxes):
            whole[(slice(None),) + tuple(slice(blo[d], bhi[d] + 1) for d in (2, 1, 0))] = \
                valid_view(lev.patch_view(flat, i), ng, 3)
        outs.append((whole, new))
        lev.close()
        ctx.close()
    assert np.array_equal(outs[0][0], outs[1][0])
    assert outs[0][1] == outs[1][1]
