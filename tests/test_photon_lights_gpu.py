"""Direct light of photon-mapped frames, by ten lanes a hit and, from 303 104 hits on, by one."""
import os

import numpy as np
import pytest

import oracle
import photon_lights
import photon_scenes
import rednoise_b200 as rn  # noqa: F401
from imgcheck import agree, argb_to_rgba, light_records
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "photon_lights.npz")


@pytest.mark.parametrize("name", sorted(photon_lights.LIGHTS))
def test_canvas_is_the_stored_one(name):
    want = np.load(GOLDEN)[name]
    assert np.array_equal(photon_lights.small(name), want)


@pytest.mark.parametrize("name", sorted(photon_lights.LIGHTS))
def test_either_side_of_the_hit_limit(name):
    """640 x 480 camera rays that all hit are 307 200 hits; the middle of the frame is the frame of
    half the size, whose camera forms the same rays exactly."""
    s = photon_scenes.scene("box")
    many, few = photon_lights.render(s, name, 640, 480), photon_lights.render(s, name, 320, 240)
    assert np.array_equal(many[120:360, 160:480], few)


@pytest.mark.skipif(not os.path.exists(oracle.REF_PATH), reason="the reference's library is not built here")
@pytest.mark.parametrize("name", sorted(photon_lights.LIGHTS))
def test_stored_canvas_matches_the_reference(name):
    if name == "three":
        pytest.skip("a scene of panes")
    box = scenes.cornell_box(light_scale=10.0)
    m = oracle.RefModel.from_arrays(np.ascontiguousarray(box["vertices"] * photon_scenes.SCALE), box["ref_rgb"],
                                    box["ref_material"], np.zeros(len(box["ref_rgb"]), np.float32))
    w, h = photon_lights.SMALL
    want = m.render_photon_mapped(w, h, 1500, lights=light_records(photon_lights.lights(name)), focal=1.2,
                                  pos=photon_lights.CAMERA["position"])
    m.close()
    agree(argb_to_rgba(np.load(GOLDEN)[name]), argb_to_rgba(want), min_equal=0.999, max_outlier_frac=0.001)
