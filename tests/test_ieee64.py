"""The integer-pipe forms of csrc/mf_ieee64.cuh against the FP64 instructions
on the GPU, bit for bit: division, square root, product, comparisons, maximum and
minimum, scaling by powers of two and minmod."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ms-flukss-multifluid_gb300", "csrc")
NAMES = ("div", "root", "compare", "maxmin", "scale", "minmod", "mul")


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = tmp_path_factory.mktemp("ieee64") / "check"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I", CSRC, os.path.join(HERE, "cuda", "ieee64_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    return dict(line.split(maxsplit=1) for line in r.stdout.strip().splitlines())


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_ieee64_equals_the_instructions(counts, name):
    assert counts["status"] == "no error"
    assert int(counts[name]) == 0
