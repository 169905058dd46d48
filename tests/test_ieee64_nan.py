"""NaN in the integer-pipe forms of csrc/mf_ieee64.cuh: maxima and comparisons
against the FP64 forms for every pair of special values."""
import os
import shutil
import subprocess

import pytest

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


@pytest.mark.parametrize("name", ["maxmin", "compare"])
def test_special_values_equal_the_fp64_forms(counts, name):
    assert counts["status"] == "no error"
    assert int(counts[name]) == 0
