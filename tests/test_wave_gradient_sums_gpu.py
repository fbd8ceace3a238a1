"""The wave adjoint's gradients at a size where the grouping of their sums shows: 8.4M samples
over 36 triangles with image gradients of one sign. Each gradient value is one float to which
every warp adds its share, and callers compare runs of these sums with each other; sums grouped
otherwise (per block, say) are other gradients. What is stored is what such chains give, not the
exact value: with terms of one sign they fall short of the sum in 64 bits, here by 1.2e-3 (0.8 %
at 128 samples a pixel, 3.4 % at 512)."""
import os

import numpy as np
import pytest

import rednoise_b200 as rn
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "wave_gradients.npz")
SIZE, SPP, DEPTH = 512, 32, 6
# A triangle's float takes up to SIZE^2 * SPP * (DEPTH - 1) / 32 = 1.3M additions, whose order changes
# from run to run: two such chains differ by about 2^-24 * sqrt(1.3M) = 7e-5 of the sum.
TOLERANCE = 1e-4


def gradients():
    room = scenes.cornell_box(light_scale=10.0)
    s = rn.Scene.from_arrays(room["vertices"], **{k: room[k] for k in ("albedo", "emission", "material",
                                                                      "material_param")})
    c = scenes.camera(SIZE, SIZE)
    cam = rn.Camera.make(c["position"], c["target"], c["up"], c["vfov_deg"], SIZE, SIZE)
    settings = rn.Settings.make(spp=SPP, max_depth=DEPTH, rr_depth=DEPTH, seed=9, integrator=2)
    return s.backward([(cam, settings)], [np.ones((SIZE, SIZE, 3), np.float32)])


def test_gradients_are_the_stored_ones():
    want = np.load(GOLDEN)
    for got, name in zip(gradients(), ("d_albedo", "d_emission")):
        w = want[name].astype(np.float64)
        assert np.linalg.norm(got - w) <= TOLERANCE * np.linalg.norm(w), name
