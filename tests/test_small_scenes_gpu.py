"""The paths that scenes with a triangle list take (a group of lanes per ray) and the row
streams' two kernels, at the sizes where they change hands: ray queries against the 2-wide
reference tree, which every query can be given, and rows against the oracle's streams."""
import numpy as np
import pytest

import oracle
import rednoise_b200 as rn
from imgcheck import agree, argb_to_rgba
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu
EXACT = dict(min_equal=0.999, max_outlier_frac=0.001)  # as the other comparisons of these streams


def _triangles(n, seed):
    """n triangles of a box and some clutter, with coplanar, repeated and degenerate ones among them."""
    rng = np.random.default_rng(seed)
    v = np.concatenate([scenes.cornell_box()["vertices"], rng.uniform(-2.5, 2.5, (max(n, 1), 9)).astype(np.float32)])[:n]
    if n > 60:
        v[50] = v[12]  # the same triangle twice
        v[51] = 0.0  # a point
        v[52, 3:6] = v[52, :3]  # a segment
    return np.ascontiguousarray(v)


def _rays(v, n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-3.0, 3.0, (n, 3)).astype(np.float32)
    w = rng.dirichlet((1.0, 1.0, 1.0), n).astype(np.float32)
    k = rng.integers(0, len(v), n)
    aim = (v[k].reshape(n, 3, 3) * w[:, :, None]).sum(1) - o  # towards points of the triangles
    d = np.where(rng.random(n)[:, None] < 0.5, aim, rng.normal(size=(n, 3))).astype(np.float32)
    corner = rng.random(n) < 0.1
    d[corner] = v[k[corner]].reshape(-1, 3, 3)[:, 0] - o[corner]
    odd = [(0, 0, -1), (1, 0, 0), (0, -0.0, 2), (1e-40, 1, 0.5), (1e30, 2e30, -1e30), (1e-30, 1e-30, 3e-30),
           (np.inf, 1, 1), (np.nan, 0, 1), (0, 0, 0)]
    m = min(n, len(odd))
    d[:m] = np.array(odd[:m], np.float32)
    return o, d, k.astype(np.int32)


@pytest.mark.parametrize("tris", [1, 4, 5, 36, 127, 128, 129])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1021])
def test_few_rays_equal_the_reference_tree(tris, n):
    v = _triangles(tris, tris)
    s = rn.Scene.from_arrays(v)
    for ignore in (None, "some"):
        o, d, k = _rays(v, n, 7 * n + tris)
        ig = None if ignore is None else k
        got, want = s.trace_closest(o, d, ig), s.trace_closest(o, d, ig, width2=True)
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        tmax = np.where(np.isfinite(want[1]), want[1] * np.float32(1.0 + 1e-6), np.float32(5.0)).astype(np.float32)
        tmax[::3] = want[1][::3]  # strictly before the hit itself: not occluded by it
        assert np.array_equal(s.trace_any(o, d, tmax, ig), s.trace_any(o, d, tmax, ig, width2=True))


@pytest.mark.parametrize("n", [65536, 65537])
def test_either_side_of_the_ray_limit(n):
    v = _triangles(36, 0)
    s = rn.Scene.from_arrays(v * np.float32(1e10))  # edges of 10^10: long directions leave the bounded test
    o, d, _ = _rays(v, n, 3)
    o = o * np.float32(1e10)
    d[100:200] *= np.float32(1e18)
    got, want = s.trace_closest(o, d), s.trace_closest(o, d, width2=True)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def _row_scene(kind):
    sc = scenes.cornell_box() if kind == "box" else scenes.icosphere_scene(2)
    return np.ascontiguousarray(sc["vertices"] * np.float32(1.0 / scenes.HALF)), sc["ref_rgb"]


@pytest.mark.parametrize("kind,w,h,spp", [("box", 1, 1, 1), ("box", 23, 9, 3), ("box", 5, 296, 2), ("box", 5, 297, 2),
                                          ("box", 320, 192, 64), ("sphere", 19, 7, 1), ("sphere", 21, 6, 2),
                                          ("sphere", 17, 6, 3), ("sphere", 9, 5, 40)])
def test_row_streams_match_the_oracle(kind, w, h, spp):
    """320 x 192 x 64 takes two chunks of columns; the oracle's rows are checked in part."""
    v, rgb = _row_scene(kind)
    s = rn.Scene.from_arrays(v, ref_rgb=rgb)
    got = s.render_bidirectional(w, h, spp, focal_length=w / 150.0, position=(0.1, 0.05, 4.0))
    y0 = max(0, h // 2 - 2)
    y1 = min(h, y0 + 4)
    want = oracle.OrcBvh(v).render_bidirectional(s.triangles()["normal"], rgb, w, h, spp, y0=y0, y1=y1,
                                                 focal=w / 150.0, pos=(0.1, 0.05, 4.0))
    agree(argb_to_rgba(got[y0:y1]), argb_to_rgba(want), **EXACT)
