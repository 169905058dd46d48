"""Options whose plasma fluxes stay in the kernel that solves every fluid
(tracking surfaces, characteristic reconstruction, HELIOBC) take the neutral
populations in a launch of their own in the FP64 paths: against the oracle with
two to five fluids, in the RK2 and the Hancock step, and their share of a
level's launch count."""
import numpy as np
import pytest

import mfgpu
from helpers import rel_err, to_device, to_host, valid_view

pytestmark = pytest.mark.gpu
N = 64
PREC = {"fp64": (mfgpu.PREC_FP64, 1e-12), "fast": (mfgpu.PREC_FP64_FAST, 1e-7)}
FORMS = {
    "tracer": dict(tracer=True),
    "tracer_positivity": dict(tracer=True, check_positivity=1),
    "char": dict(char_reconstruction=1),
    "char_positivity": dict(char_reconstruction=1, check_positivity=1),
    "heliobc": dict(helio_bc=1),
    "heliobc_tracer": dict(tracer=True, helio_bc=1),
}


def _params(form, nf, glm, prec, ta, n=N):
    kw = dict(FORMS[form])
    p = mfgpu.helio_params(n, region_tracer=kw.pop("tracer", False), precision=prec,
                           time_approximation=ta)
    p.n_fluids = nf
    p.charge_exchange = p.neutral_sun_bc = int(nf > 1)
    if not glm:
        p.divb_cleaning, p.use_8wave = 0, 1
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def _state(p, glm, lo, hi, n=N):
    U = mfgpu.init_host_fab(mfgpu.helio_params(n), lo, hi, "helio")
    U = U * (1.0 + 0.02 * np.random.default_rng(5).standard_normal(U.shape))
    parts = [U[: 9 if glm else 8]] + [U[9 + 5 * (f % 3) : 14 + 5 * (f % 3)]
                                      for f in range(p.n_fluids - 1)]
    if p.num_tracking_surfaces:  # between the regions, as a run has it after some steps
        parts.append(np.tanh(np.random.default_rng(6).standard_normal(U[:1].shape)))
    return np.ascontiguousarray(np.concatenate(parts))


@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("ta", [mfgpu.TA_RK2, mfgpu.TA_HANCOCK], ids=["rk2", "hancock"])
@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("nf,glm,size", [(2, True, (1, 1, 1)), (3, False, (13, 5, 2)),
                                         (4, True, (9, 7, 4)), (5, False, (7, 11, 3))])
def test_apart_equals_oracle(gpulib, oracle, prec, ta, form, nf, glm, size):
    code, tol = PREC[prec]
    p = _params(form, nf, glm, code, ta)
    q = _params(form, nf, glm, mfgpu.PREC_FP64, ta)
    vlo = [0, 30, N - size[2]] if "heliobc" in form else [46, 30, 29]  # at two sides of the domain
    vhi = [vlo[d] + size[d] - 1 for d in range(3)]
    lo, hi = mfgpu.grow(vlo, vhi, mfgpu.num_ghost(p), 3)
    U = _state(p, glm, lo, hi)
    dt = 0.1 * oracle.compute_dt(q, U, lo, hi, vlo, vhi)[1]
    ctx = mfgpu.Context(p)
    t = to_device(U)
    _, ndt, _ = ctx.patch_update(t.data_ptr(), lo, hi, vlo, vhi, dt)
    g = valid_view(to_host(t), ctx.ng, 3)
    ctx.close()
    st, ndto, _ = oracle.patch_update(q, U, lo, hi, vlo, vhi, dt)
    assert st == 0
    err = rel_err(g, valid_view(U, mfgpu.num_ghost(p), 3))
    assert np.all(err <= tol), err
    assert abs(ndt - ndto) <= tol * ndto


@pytest.mark.parametrize("prec", sorted(PREC))
@pytest.mark.parametrize("ta,stages", [(mfgpu.TA_RK2, 2), (mfgpu.TA_HANCOCK, 1)])
@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("nf", [1, 4])
def test_apart_launches_are_counted(gpulib, prec, ta, stages, form, nf):
    n = 16
    p = _params(form, nf, True, PREC[prec][0], ta, n)
    apart = nf > 1 and (ta == mfgpu.TA_HANCOCK or form != "char_positivity")
    ctx = mfgpu.Context(p)
    lev = mfgpu.Level(ctx, mfgpu.tile_boxes(n, 8, 3))
    buf = np.zeros(lev.ndoubles)
    for i in range(len(lev.boxes)):
        lev.patch_view(buf, i)[:] = _state(p, True, *lev.fab_box(i), n)
    lev.upload(buf.ctypes.data)
    prof = lev.profile_step(0.05 * lev.compute_dt()[0])
    assert len(prof) == lev.launches_per_step()
    assert sum(k == "flux" for k, _ in prof) == stages * (3 + apart)
    lev.close()
    ctx.close()
