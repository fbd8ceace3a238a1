"""The bidirectional renderer's row streams over scenes without a triangle list, around the number
of samples at which their kernel changes: random triangles that share their leaves' boxes, with
repeated and degenerate ones among them, against the oracle's streams."""
import numpy as np
import pytest

import oracle
import rednoise_b200 as rn
from imgcheck import agree, argb_to_rgba
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris,w,h,spp", [(129, 13, 5, 3), (129, 13, 5, 4), (3000, 24, 6, 1), (3000, 7, 300, 3),
                                          (3001, 9, 5, 4)])
def test_row_streams_match_the_oracle(tris, w, h, spp):
    rng = np.random.default_rng(tris)
    room = scenes.cornell_box()["vertices"] * np.float32(1.0 / scenes.HALF)
    at = rng.uniform(-0.9, 0.9, (tris - len(room), 1, 3))
    soup = (at + rng.normal(size=(len(at), 3, 3)) * 0.1).reshape(-1, 9).astype(np.float32)
    soup[3] = soup[2]
    soup[4] = np.tile(soup[4, :3], 3)
    v = np.ascontiguousarray(np.concatenate([room, soup]))
    rgb = rng.integers(60, 220, (tris, 3)).astype(np.int32)
    s = rn.Scene.from_arrays(v, ref_rgb=rgb)
    got = s.render_bidirectional(w, h, spp, focal_length=w / 150.0, position=(0.1, 0.05, 4.0))
    y0 = max(0, h // 2 - 2)
    y1 = min(h, y0 + 4)
    want = oracle.OrcBvh(v).render_bidirectional(s.triangles()["normal"], rgb, w, h, spp, y0=y0, y1=y1,
                                                 focal=w / 150.0, pos=(0.1, 0.05, 4.0))
    # as the other comparisons of these streams
    agree(argb_to_rgba(got[y0:y1]), argb_to_rgba(want), min_equal=0.999, max_outlier_frac=0.001)
