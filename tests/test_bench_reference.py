"""bench.py where the reference's library is not built: its arm says so on one line, and what it
would be compared with is marked, not missing. CPU only."""
import json
import os
import subprocess
import sys

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_its_library(tmp_path):
    """A copy of the two files that the arm needs, beside no library."""
    os.makedirs(tmp_path / "oracle")
    for f in ("bench.py", os.path.join("oracle", "__init__.py")):
        with open(os.path.join(ROOT, f), "rb") as a, open(tmp_path / f, "wb") as b:
            b.write(a.read())
    os.symlink(os.path.join(ROOT, "rednoise_b200"), tmp_path / "rednoise_b200")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference"], cwd=tmp_path, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and line["unavailable"]


def test_cpu_baseline_without_its_library(monkeypatch):
    import bench

    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    assert bench.cpu_baseline(None)["unavailable"]
    assert bench.reference_frame(None, None, "")[1]["unavailable"]
