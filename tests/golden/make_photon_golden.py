"""Writes the photon mapper's stored canvases (needs the GPU): photon_canvases.npz of
tests/photon_scenes.py, photon_lanes.npz of tests/test_photon_lanes_gpu.py and photon_lights.npz of
tests/photon_lights.py. They are those of the build of commit 991876a, whose photon mapper shaded a
pixel per thread and was compared with the reference's own; RN_B200_LIBRARY names that build."""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path[:0] = [ROOT, os.path.join(ROOT, "tests")]
import photon_lights  # noqa: E402
import photon_scenes  # noqa: E402
import test_photon_lanes_gpu  # noqa: E402

if __name__ == "__main__":
    out = sys.argv[1] if len(sys.argv) > 1 else os.path.join(ROOT, "tests", "golden")
    canvases = {}
    for name in photon_scenes.FRAMES:
        canvas, stored = photon_scenes.render(name)
        canvases[name], canvases[name + "_stored"] = canvas, np.int64(stored)
    np.savez_compressed(os.path.join(out, "photon_canvases.npz"), **canvases)
    np.savez_compressed(os.path.join(out, "photon_lanes.npz"),
                        **{n: test_photon_lanes_gpu.render(n) for n in test_photon_lanes_gpu.FRAMES})
    np.savez_compressed(os.path.join(out, "photon_lights.npz"),
                        **{n: photon_lights.small(n) for n in photon_lights.LIGHTS})
