"""What photon-mapped frames ask for: with a final gather nothing per pixel but the canvas, and
without one a frame whose list of diffuse hits finds no room is made with a short list."""
import ctypes

import numpy as np
import pytest
import torch

import photon_scenes
from rednoise_b200 import _native

pytestmark = pytest.mark.gpu


def _render(s, w, h, gather=0):
    return s.render_photon_mapped(w, h, 500, gather_rays=gather, position=(0.05, 0.1, 4.0),
                                  focal_length=2.0 * h / 240.0)


def test_final_gather_keeps_no_list_of_hits():
    s = photon_scenes.scene("box")
    _render(s, 8, 8, 1)  # the kernels are loaded
    free = torch.cuda.mem_get_info()[0]
    _render(s, 1024, 512, 1)
    # 500 photons and a canvas of 2 MB; a list of two hits a pixel would take 88 MB
    assert free - torch.cuda.mem_get_info()[0] < 16 << 20


# 2^18 hits are kept when memory is short: bands of rows, and strips of 2^14 columns
@pytest.mark.parametrize("size", [(640, 480), (20000, 8)])
def test_frame_without_room_for_its_hits(size):
    s = photon_scenes.scene("panes")
    want = _render(s, *size)
    s.close()
    s = photon_scenes.scene("panes")
    s.prepare()
    lib = _native.load()
    lib.rn_pt_inject_allocation_failure(ctypes.c_longlong(0))
    try:
        got = _render(s, *size)
    finally:
        lib.rn_pt_inject_allocation_failure(ctypes.c_longlong(-1))
    assert np.array_equal(got, want)
