"""The photon mapper's stages at the sizes where they can go wrong: canvases and photon counts
equal the stored ones exactly (every sum is formed in the reference's order)."""
import os

import numpy as np
import pytest

import photon_scenes

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "photon_canvases.npz")


@pytest.mark.parametrize("name", sorted(photon_scenes.FRAMES))
def test_canvas_is_the_stored_one(name):
    want = np.load(GOLDEN)
    canvas, stored = photon_scenes.render(name)
    assert stored == int(want[name + "_stored"])
    assert np.array_equal(canvas, want[name])
