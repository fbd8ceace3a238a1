"""The traversal's device code compiles without warnings: a result read beside the call that
sets it (nvcc's 549-D) is one of the faults that only a warning shows. CPU only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rednoise_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no CUDA compiler")
@pytest.mark.parametrize("source", ["trace_kernels.cu", "gi.cu"])
def test_no_warnings(source, tmp_path):
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++20", "-Xptxas", "-O0",
                        "--expt-relaxed-constexpr", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-c",
                        os.path.join(CSRC, source), "-o", str(tmp_path / "out.o")], capture_output=True, text=True)
    assert r.returncode == 0 and "warning" not in r.stderr, r.stderr[-3000:]
