"""Photon-mapped frames with more gathers than get a block each: those by lanes, which leave out
the photons that are too far from all points of their warp, give the stored canvases exactly."""
import os

import numpy as np
import pytest

import photon_scenes
import rednoise_b200 as rn  # noqa: F401

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "photon_lanes.npz")
# name: (scene, width, height, photons); 148 * 64 = 9472 gathers have a block each
FRAMES = {
    "just_past": ("box", 137, 101, 3000),
    "room": ("box", 240, 181, 6000),
    "mesh": ("sphere", 211, 163, 6000),
    "panes": ("panes", 160, 120, 1500),
}


def render(name):
    kind, w, h, photons = FRAMES[name]
    return photon_scenes.scene(kind).render_photon_mapped(w, h, photons, position=(0.05, 0.1, 4.0),
                                                          focal_length=2.0 * h / 240.0)


@pytest.mark.parametrize("name", sorted(FRAMES))
def test_canvas_is_the_stored_one(name):
    want = np.load(GOLDEN)[name]
    assert np.array_equal(render(name), want)
