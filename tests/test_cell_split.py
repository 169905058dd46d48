"""The update with one thread per cell and fluid (mf_cell_kernel.cuh) against
the oracle: one to five fluids, with GLM cleaning or the 8-wave source, with
and without charge exchange, in patches of one cell and around a block's 64
cells (one block exactly, one cell less and more, several blocks), half of
them across the edge of the reset sphere; and the levels' own ghost copies and
far-field fill, which leave the edges and corners of the ghost layers alone."""
import numpy as np
import pytest

import mfgpu
from helpers import rel_err, to_device, to_host, valid_view

pytestmark = pytest.mark.gpu
RTOL = 1e-12  # per step and conserved variable, the parity path's bar

N = 64
SIZES = [(1, 1, 1), (4, 4, 4), (7, 9, 1), (13, 5, 1), (9, 7, 4)]


def _params(nf, glm, ce):
    p = mfgpu.helio_params(N)
    p.n_fluids = nf
    p.charge_exchange = int(ce and nf > 1)
    p.neutral_sun_bc = int(nf > 1)
    if not glm:
        p.divb_cleaning, p.use_8wave = 0, 1
    return p


def _state(p, nf, glm, lo, hi):
    U = mfgpu.init_host_fab(mfgpu.helio_params(N), lo, hi, "helio")
    rng = np.random.default_rng(11)
    U = U * (1.0 + 0.02 * rng.standard_normal(U.shape))
    plasma, neutral = U[: 9 if glm else 8], U[9:]
    parts = [plasma] + [neutral[5 * (f % 3) : 5 * (f % 3) + 5] for f in range(nf - 1)]
    return np.ascontiguousarray(np.concatenate(parts))


@pytest.mark.parametrize("nf,glm,ce", [(1, True, False), (2, True, True), (3, False, True),
                                       (4, True, True), (4, False, False), (5, True, True)])
@pytest.mark.parametrize("size", SIZES)
def test_update_by_fluid_equals_oracle(gpulib, oracle, nf, glm, ce, size):
    p = _params(nf, glm, ce)
    ctx = mfgpu.Context(p)
    vlo = [34, 30, 29]
    vhi = [vlo[d] + size[d] - 1 for d in range(3)]
    lo, hi = mfgpu.grow(vlo, vhi, ctx.ng, 3)
    U = _state(p, nf, glm, lo, hi)
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


@pytest.mark.parametrize("nf", [1, 4, 5])
@pytest.mark.parametrize("n,patch", [(12, 6), (20, 10), (22, 11)])
def test_level_ghosts_equal_single_patches(gpulib, nf, n, patch):
    """A level's step (primitive copies and far-field ghosts on the faces of
    the ghost layers) equals the step of one patch that holds the whole domain
    bitwise, far-field boundary included."""
    outs = []
    for size in (patch, n):
        p = mfgpu.helio_params(n)
        p.n_fluids = nf
        p.charge_exchange = p.neutral_sun_bc = int(nf > 1)
        ctx = mfgpu.Context(p)
        lev = mfgpu.Level(ctx, mfgpu.tile_boxes(n, size, 3))
        flat = np.zeros(lev.ndoubles)
        for i in range(len(lev.boxes)):
            lo, hi = lev.fab_box(i)
            full = _domain_state(n, nf)
            lev.patch_view(flat, i)[:] = full[(slice(None),) + tuple(
                slice(lo[d] + ctx.ng, hi[d] + ctx.ng + 1) for d in (2, 1, 0))]
        lev.upload(flat.ctypes.data)
        dt = 0.2 * lev.compute_dt()[0]
        for _ in range(2):
            st, _, _, _ = lev.step(dt)
            assert st == 0
        lev.download(flat.ctypes.data)
        whole = np.zeros((lev.patch_view(flat, 0).shape[0], n, n, n))
        for i, (blo, bhi) in enumerate(lev.boxes):
            whole[(slice(None),) + tuple(slice(blo[d], bhi[d] + 1) for d in (2, 1, 0))] = \
                valid_view(lev.patch_view(flat, i), ctx.ng, 3)
        outs.append(whole)
        lev.close()
    assert np.array_equal(outs[0], outs[1])


def _domain_state(n, nf):
    p = mfgpu.helio_params(n)
    ng = mfgpu.Context(p).ng
    U = mfgpu.init_host_fab(p, [-ng] * 3, [n - 1 + ng] * 3, "helio")
    U = U * (1.0 + 0.01 * np.random.default_rng(3).standard_normal(U.shape))
    parts = [U[:9]] + [U[9 + 5 * (f % 3) : 14 + 5 * (f % 3)] for f in range(nf - 1)]
    return np.concatenate(parts)
