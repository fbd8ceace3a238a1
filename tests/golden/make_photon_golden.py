"""Writes photon_canvases.npz, the photon mapper's canvases of tests/photon_scenes.py (needs the GPU);
photon_lanes.npz holds those of tests/test_photon_lanes_gpu.py from the same build. Kept from the build whose photon mapper was checked against the reference's own."""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path[:0] = [ROOT, os.path.join(ROOT, "tests")]
import photon_scenes  # noqa: E402

if __name__ == "__main__":
    out = {}
    for name in photon_scenes.FRAMES:
        canvas, stored = photon_scenes.render(name)
        out[name], out[name + "_stored"] = canvas, np.int64(stored)
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else os.path.join(ROOT, "tests", "golden",
                                                                          "photon_canvases.npz"), **out)
