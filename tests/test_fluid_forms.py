"""The kernels split by fluid in the forms that the parity path's RK2 step does
not reach, against the oracle: fast FP64 and mixed precision, the Hancock
predictor and corrector, one to five fluids; the positivity fallback of the
face fluxes where it fires; the no-allocation call of a patch that leaves no
room for the update by fluid; and the fast FP64 fluxes by lines, which round
as those per face."""
import ctypes

import numpy as np
import pytest

import mfgpu
from helpers import component_groups, rel_err, to_device, to_host, valid_view

pytestmark = pytest.mark.gpu
N = 64
FLUIDS = [(1, True, False), (2, True, True), (3, False, True), (4, True, True), (4, False, False),
          (5, True, True)]


def _params(nf, glm, ce, **kw):
    p = mfgpu.helio_params(N, **kw)
    p.n_fluids = nf
    p.charge_exchange = int(ce and nf > 1)
    p.neutral_sun_bc = int(nf > 1)
    if not glm:
        p.divb_cleaning, p.use_8wave = 0, 1
    return p


def _state(nf, glm, lo, hi, seed=11):
    U = mfgpu.init_host_fab(mfgpu.helio_params(N), lo, hi, "helio")
    U = U * (1.0 + 0.02 * np.random.default_rng(seed).standard_normal(U.shape))
    parts = [U[: 9 if glm else 8]] + [U[9 + 5 * (f % 3) : 14 + 5 * (f % 3)] for f in range(nf - 1)]
    return np.ascontiguousarray(np.concatenate(parts))


def _boxes(p, size, vlo=(34, 30, 29)):
    vlo = list(vlo)
    vhi = [vlo[d] + size[d] - 1 for d in range(3)]
    return vlo, vhi, *mfgpu.grow(vlo, vhi, mfgpu.num_ghost(p), 3)


def _step(p, U, box, dt):
    vlo, vhi, lo, hi = box
    ctx = mfgpu.Context(p)
    t = to_device(U)
    _, ndt, cell = ctx.patch_update(t.data_ptr(), lo, hi, vlo, vhi, dt)
    out = valid_view(to_host(t), ctx.ng, 3)
    ctx.close()
    return out, ndt, cell


def _group_err(a, b):
    """Mean and largest |a - b| of each component over the largest value of its
    group."""
    out = np.zeros((2, b.shape[0]))
    for g in component_groups(b.shape[0]):
        s = np.max(np.abs(b[g]))
        for c in g:
            d = np.abs(a[c] - b[c]) / s
            out[:, c] = d.mean(), d.max()
    return out


@pytest.mark.parametrize("ta", [mfgpu.TA_RK2, mfgpu.TA_HANCOCK], ids=["rk2", "hancock"])
@pytest.mark.parametrize("prec", ["fp64", "fast", "mixed"])
@pytest.mark.parametrize("nf,glm,ce", FLUIDS)
@pytest.mark.parametrize("size", [(1, 1, 1), (13, 5, 1), (9, 7, 4)])
def test_forms_equal_oracle(gpulib, oracle, ta, prec, nf, glm, ce, size):
    """fp64: 1e-12 as everywhere.  fast: 1e-7, the square root of epsilon near
    the Roe solver's triple point.  mixed: a step moves a value by the face
    fluxes times dt/dx, at a CFL number of 0.2 by a fraction of the value,
    with the FP32 solver's rounding: a few tens of 2^-24 on average, the root
    of 2^-24 near the triple point; psi starts from the state's 2 % noise in
    B, which makes its own values 50 times smaller than the terms they come
    from."""
    code = dict(fp64=mfgpu.PREC_FP64, fast=mfgpu.PREC_FP64_FAST, mixed=mfgpu.PREC_MIXED)[prec]
    p = _params(nf, glm, ce, time_approximation=ta, precision=code)
    q = _params(nf, glm, ce, time_approximation=ta)
    # (mixed: off the wind sphere, at whose edge the FP32 fluxes of cold plasma
    # are Rusanov's)
    box = _boxes(p, size, (48, 47, 45) if prec == "mixed" else (34, 30, 29))
    U = _state(nf, glm, box[2], box[3])
    dt = 0.2 * oracle.compute_dt(q, U, box[2], box[3], box[0], box[1])[1]
    g, ndt, cell = _step(p, U, box, dt)
    st, ndto, cello = oracle.patch_update(q, U, box[2], box[3], box[0], box[1], dt)
    assert st == 0
    o = valid_view(U, mfgpu.num_ghost(p), 3)
    if prec == "mixed":
        mean, most = _group_err(g, o)
        psi = np.arange(len(o)) == (8 if glm else -1)
        assert np.all(mean <= np.where(psi, 5e-4, 1e-5)), mean
        assert np.all(most <= np.where(psi, 5e-4, 2.5e-4)), most
        assert abs(ndt - ndto) <= 2.5e-4 * ndto
        return
    tol = 1e-12 if prec == "fp64" else 1e-7
    err = rel_err(g, o)
    assert np.all(err <= tol), err
    assert abs(ndt - ndto) <= tol * ndto
    if prec == "fp64":
        assert cell == cello


def _step_down(U, at):
    """Density and pressure lower in the octant from cell at on, by 20, and by
    10 again from the next cell on."""
    U[:5, at:, at:, at:] /= 20.0
    U[:5, at + 1 :, at + 1 :, at + 1 :] /= 10.0
    return U


@pytest.mark.parametrize("prec", ["fp64", "fast"])
@pytest.mark.parametrize("nf,glm", [(1, True), (4, True), (3, False)])
def test_positivity_fallback_fires(gpulib, oracle, prec, nf, glm):
    """The hyperbee slopes of rho and p leave the neighbours' range between two
    steep drops and put face values below zero in every direction; those cells
    take their own value on their faces, in every fluid."""
    code = dict(fp64=mfgpu.PREC_FP64, fast=mfgpu.PREC_FP64_FAST)[prec]
    p = _params(nf, glm, True, precision=code)
    q = _params(nf, glm, True)
    for r in (p, q):
        r.check_positivity = 1
        r.limiter[0] = r.limiter[4] = mfgpu.LIM_HYPERBEE
    box = _boxes(p, (9, 9, 9), (48, 47, 45))
    U = _step_down(_state(nf, glm, box[2], box[3]), 8)
    rho = U[0]
    pres = (p.gamma - 1.0) * (U[4] - 0.5 * (U[1:4] ** 2).sum(0) / rho
                              - (U[5:8] ** 2).sum(0) / (8.0 * np.pi))
    assert rho.min() > 0 and pres.min() > 0
    for w in (rho, pres):
        for d in range(3):  # cell 8 along d, inside the octant across it
            x = [w[tuple(9 if e != d else 8 + o for e in range(3))] for o in (-1, 0, 1)]
            assert min(oracle.face_values(mfgpu.LIM_HYPERBEE, *x)) <= 0.0
    dt = 0.1 * oracle.compute_dt(q, U, box[2], box[3], box[0], box[1])[1]
    g, ndt, cell = _step(p, U, box, dt)
    st, ndto, cello = oracle.patch_update(q, U, box[2], box[3], box[0], box[1], dt)
    assert st == 0
    tol = 1e-12 if prec == "fp64" else 1e-7
    err = rel_err(g, valid_view(U, mfgpu.num_ghost(p), 3))
    assert np.all(err <= tol), err
    assert abs(ndt - ndto) <= tol * ndto
    if prec == "fp64":
        assert cell == cello


def _scratch(size, nc, bytes_per_flux, cells_per_partial):
    """Bytes of the static array that an RK2 call of an interior patch takes."""
    up = lambda x: (x + 255) // 256 * 256  # noqa: E731
    prod = lambda b: b[0] * b[1] * b[2]  # noqa: E731
    total = 2 * up(8 * nc * prod([s + 8 for s in size]))
    for g in (4, 0):
        for d in range(3):
            n = prod([s + g + (e == d) for e, s in enumerate(size)])
            total += up(bytes_per_flux * nc * n) + up(bytes_per_flux * n)
    total += 768 + 256  # descriptors and run parameters, step state
    return total + up(16 * ((prod(size) + cells_per_partial - 1) // cells_per_partial + 1))


@pytest.mark.parametrize("prec,nf,size", [("fp64", 2, (18, 22, 27)), ("fp64", 5, (5, 11, 59)),
                                          ("mixed", 4, (10, 26, 32)), ("mixed", 1, (28, 28, 36))])
def test_noalloc_without_room_for_finer_partials(gpulib, prec, nf, size):
    """Patches that fill the scratch array to its last kilobyte: room for one
    time-step partial per 128 cells, none for one per 64."""
    code = dict(fp64=mfgpu.PREC_FP64, mixed=mfgpu.PREC_MIXED)[prec]
    p = _params(nf, True, True, precision=code)
    ctx = mfgpu.Context(p)
    rs = 4 if prec == "mixed" else 8
    assert _scratch(size, ctx.nc, rs, 128) <= mfgpu.NOALLOC_SCRATCH_BYTES
    assert _scratch(size, ctx.nc, rs, 64) > mfgpu.NOALLOC_SCRATCH_BYTES
    vlo, vhi, lo, hi = _boxes(p, size, [s if s + e < 60 else 2 for s, e in zip((20, 18, 15), size)])
    U = _state(nf, True, lo, hi)
    res = []
    for fn in (ctx.lib.mf_patch_update, ctx.lib.mf_patch_update_noalloc):
        t = to_device(U)
        fab = mfgpu.MfFab(t.data_ptr(), mfgpu.make_box(lo, hi), ctx.nc)
        valid = mfgpu.make_box(vlo, vhi)
        ndt, cell = ctypes.c_double(), mfgpu.c_int3()
        st = fn(ctx.h, ctypes.byref(fab), ctypes.byref(valid), 2e-4, None, None,
                ctypes.byref(ndt), cell, None)
        assert st == mfgpu.MF_OK
        res.append((valid_view(to_host(t), ctx.ng, 3), ndt.value, tuple(cell)))
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1:] == res[1][1:]
    ctx.close()


@pytest.mark.parametrize("form", ["helio", "char", "heliobc", "rusanov", "vfroe", "orszag"])
def test_fast_lines_equal_faces_bitwise(gpulib, form):
    """Every product that the fast FP64 fluxes fuse is written out, so the
    kernels of both forms give the same bits."""
    n, patch, sd, init = (32, 16, 3, "helio") if form != "orszag" else (64, 16, 2, "orszag")
    if form == "orszag":
        p = mfgpu.orszag_params(n, precision=mfgpu.PREC_FP64_FAST)
    else:
        p = mfgpu.helio_params(n, precision=mfgpu.PREC_FP64_FAST, region_tracer=form == "heliobc")
        p.char_reconstruction = int(form == "char")
        p.helio_bc = int(form == "heliobc")
        if form in ("rusanov", "vfroe"):
            p.divb_cleaning, p.use_8wave, p.flux = 0, 1, 2 if form == "rusanov" else 5
    ctx = mfgpu.Context(p)
    lev = mfgpu.Level(ctx, mfgpu.tile_boxes(n, patch, sd))
    buf = np.zeros(lev.ndoubles)
    for i in range(len(lev.boxes)):
        lev.patch_view(buf, i)[:] = mfgpu.init_host_fab(p, *lev.fab_box(i), init)
    res = []
    for which in (mfgpu.FLUX_FACES, mfgpu.FLUX_LINES):
        lev.upload(buf.ctypes.data)
        lev.set_time(0.0)
        lev.set_flux_form(which)
        dt = 0.4 * lev.compute_dt()[0]
        steps = []
        for _ in range(2):
            st, nd, ip, cell = lev.step(dt)
            steps.append((st, nd, ip, cell))
            dt = 0.4 * nd
        out = np.zeros(lev.ndoubles)
        lev.download(out.ctypes.data)
        res.append((out, steps))
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1] == res[1][1]
    lev.close()
    ctx.close()
