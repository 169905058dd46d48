"""The FP64 face fluxes with the plasma and the neutral populations in
launches of their own, all directions in one (mf_face_kernel.cuh), against the
oracle: every solver, averaging and limiter kind that the kernels take, with
and without the positivity fallback, in patch sizes around a block's 64 and
128 faces (one cell wide, odd, several blocks per direction), and their share
of a level's launch count."""
import numpy as np
import pytest

import mfgpu
from helpers import rel_err, to_device, to_host, valid_view

pytestmark = pytest.mark.gpu
RTOL = 1e-12  # per step and conserved variable, the parity path's bar

PLAIN = dict(divb_cleaning=0, use_8wave=1)
FORMS = {
    "glm": dict(flux=1),
    "glm_roe_average": dict(flux=3),
    "roe8": dict(PLAIN, flux=1),
    "roe7_roe_average": dict(PLAIN, flux=13),
    "rusanov": dict(PLAIN, flux=2),
    "vfroe": dict(PLAIN, flux=5),
    "limiters_positivity": dict(flux=1, limiters=True, check_positivity=1),
    "central_bn": dict(PLAIN, flux=1, divb_method=2),
}


def _params(form):
    p = mfgpu.helio_params(64)
    for k, v in FORMS[form].items():
        if k == "limiters":
            for q in range(8):
                p.limiter[q] = (mfgpu.LIM_VANLEER, mfgpu.LIM_MC, mfgpu.LIM_MINMOD)[q % 3]
        else:
            setattr(p, k, v)
    return p


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("size", [(1, 1, 1), (3, 5, 2), (9, 7, 4)])
def test_split_fluxes_equal_oracle(gpulib, oracle, form, size):
    p = _params(form)
    ctx = mfgpu.Context(p)
    vlo = [34, 30, 29]
    vhi = [vlo[d] + size[d] - 1 for d in range(3)]
    lo, hi = mfgpu.grow(vlo, vhi, ctx.ng, 3)
    rng = np.random.default_rng(7)
    U = mfgpu.init_host_fab(p, lo, hi, "helio")
    U *= 1.0 + 0.02 * rng.standard_normal(U.shape)
    st, dt0, _ = oracle.compute_dt(p, U, lo, hi, vlo, vhi)
    assert st == 0
    dt = 0.2 * dt0
    t = to_device(U)
    _, ndt, cell = ctx.patch_update(t.data_ptr(), lo, hi, vlo, vhi, dt)
    Uo = U.copy()
    st, ndto, cello = oracle.patch_update(p, Uo, lo, hi, vlo, vhi, dt)
    assert st == 0
    err = rel_err(valid_view(to_host(t), ctx.ng, 3), valid_view(Uo, ctx.ng, 3))
    assert np.all(err <= RTOL), err
    assert abs(ndt - ndto) <= RTOL * ndto and cell == cello


@pytest.mark.parametrize("prec", [mfgpu.PREC_FP64, mfgpu.PREC_FP64_FAST])
def test_split_launches_are_counted(gpulib, prec):
    n = 16
    for p, init, sd, flux in ((mfgpu.helio_params(n, precision=prec), "helio", 3, 2),
                              (mfgpu.orszag_params(n, precision=prec), "orszag", 2, 1)):
        ctx = mfgpu.Context(p)
        lev = mfgpu.Level(ctx, mfgpu.tile_boxes(n, 8, sd))
        buf = np.zeros(lev.ndoubles)
        for i in range(len(lev.boxes)):
            lev.patch_view(buf, i)[:] = mfgpu.init_host_fab(p, *lev.fab_box(i), init)
        lev.upload(buf.ctypes.data)
        dt = 0.2 * lev.compute_dt()[0]
        for form, per in ((mfgpu.FLUX_FACES, flux), (mfgpu.FLUX_LINES, sd)):
            lev.set_flux_form(form)
            prof = lev.profile_step(dt)
            assert len(prof) == lev.launches_per_step()
            assert sum(k == "flux" for k, _ in prof) == 2 * per
