"""NaN in the integer-pipe forms of csrc/mf_ieee64.cuh: minmod, maxima and
comparisons against the FP64 forms for every pair of special values; and a
step beside a cell that holds NaN, whose neighbours' slopes come from the
finite difference alone."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import mfgpu
from helpers import to_device, to_host

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ms-flukss-multifluid_gb300", "csrc")


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = tmp_path_factory.mktemp("ieee64_nan") / "check"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I", CSRC, os.path.join(HERE, "cuda", "ieee64_nan_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    return dict(line.split(maxsplit=1) for line in r.stdout.strip().splitlines())


@pytest.mark.parametrize("name", ["minmod", "maxmin", "compare"])
def test_special_values_equal_the_fp64_forms(counts, name):
    assert counts["status"] == "no error"
    assert int(counts[name]) == 0


@pytest.mark.parametrize("prec", [mfgpu.PREC_FP64, mfgpu.PREC_FP64_FAST])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_second_cell_beside_nan_equals_oracle(gpulib, oracle, prec, axis):
    """One first-order step with one NaN cell c: cell c+2 along axis is
    reached by c through the limiter of c+1 alone."""
    n = 9
    p = mfgpu.helio_params(64, time_approximation=mfgpu.TA_FIRST_ORDER, precision=prec)
    ctx = mfgpu.Context(p)
    vlo = [34, 30, 29]
    vhi = [v + n - 1 for v in vlo]
    lo, hi = mfgpu.grow(vlo, vhi, ctx.ng, 3)
    U = mfgpu.init_host_fab(p, lo, hi, "helio")
    U *= 1.0 + 0.02 * np.random.default_rng(9).standard_normal(U.shape)
    dt = 0.2 * oracle.compute_dt(p, U, lo, hi, vlo, vhi)[1]
    c = [ctx.ng + 3] * 3  # (z, y, x) in the fab
    U[(slice(None), *c)] = np.nan
    t = to_device(U)
    st, _, _ = ctx.patch_update(t.data_ptr(), lo, hi, vlo, vhi, dt, allow_error=True)
    assert st == mfgpu.MF_ERR_NONFINITE
    oracle.patch_update(p, U, lo, hi, vlo, vhi, dt)
    at = list(c)
    at[2 - axis] += 2
    g, o = to_host(t)[(slice(None), *at)], U[(slice(None), *at)]
    assert np.all(np.isfinite(o))
    scale = np.maximum(np.abs(o), 1e-3 * np.max(np.abs(U[:, ctx.ng, ctx.ng, ctx.ng])))
    assert np.all(np.abs(g - o) <= (1e-12 if prec == mfgpu.PREC_FP64 else 1e-7) * scale)
    ctx.close()
