"""tests/host_threads.cpp: preparing a scene where threads cannot be had. CPU only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_trees_without_threads(tmp_path):
    exe = str(tmp_path / "host_threads")
    subprocess.run(["g++", "-std=c++20", "-O2", "-I" + os.path.join(ROOT, "rednoise_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "host_threads.cpp"),
                    os.path.join(ROOT, "rednoise_b200", "csrc", "host_scene.cpp"), "-o", exe, "-pthread", "-ldl"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "thread checks passed" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
