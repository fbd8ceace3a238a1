"""tests/host_tree.cpp built with the BVH builder under AddressSanitizer + UndefinedBehaviorSanitizer. CPU only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_tree_over_the_reference_leaves(tmp_path):
    exe = str(tmp_path / "host_tree")
    subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                    "-I" + os.path.join(ROOT, "rednoise_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "host_tree.cpp"),
                    os.path.join(ROOT, "rednoise_b200", "csrc", "host_scene.cpp"), "-o", exe, "-pthread"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "tree checks passed" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
