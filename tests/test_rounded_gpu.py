"""The branch-free reciprocal and square root (rounded.cuh) on every float of their ranges, the forms
for any argument and a ray's reciprocals on every float: the bits of CUDA's correctly rounded
operations. Built here with the compiler and the options of the library."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no CUDA compiler")
@pytest.mark.parametrize("options", [[], ["-fmad=false"]])
def test_results_are_correctly_rounded(options, tmp_path):
    exe = str(tmp_path / "rounded_check")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++20", "-O3",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "rednoise_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), *options, os.path.join(ROOT, "tests", "rounded_check.cu"),
                    "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-500:] + r.stderr[-2000:]
