"""Queries over the traversal tree (the reference's leaves under boxes of their own) against the
2-wide reference tree, which WIDTH2 queries walk node by node: hits and occlusion bit for bit."""
import numpy as np
import pytest

import rednoise_b200 as rn
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu


def _vertices(kind):
    rng = np.random.default_rng(3)
    if kind == "room":
        return scenes.icosphere_scene(5)["vertices"]
    n = {"mixed": 5000, "chain": 3000, "stack": 2000, "just_past_the_list": 129}[kind]
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    size = 10.0 ** rng.uniform(-3.0, 0.5, (n, 1, 1))
    if kind == "chain":  # each triangle larger and farther than the last
        size = 1.4 ** (np.arange(n) % 120)[:, None, None]
        c = c * size
    if kind == "stack":  # parallel sheets: many equal entry distances and hits
        c = np.round(c * 4.0) / 4.0
        v = c + np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]]) * 0.5
        return v.reshape(-1, 9).astype(np.float32)
    return (c + size * rng.uniform(-1.0, 1.0, (n, 3, 3))).reshape(-1, 9).astype(np.float32)


@pytest.mark.parametrize("kind", ["room", "mixed", "chain", "stack", "just_past_the_list"])
def test_hits_equal_the_reference_tree(kind):
    v = np.ascontiguousarray(_vertices(kind), np.float32)
    s = rn.Scene.from_arrays(v)
    rng = np.random.default_rng(11)
    n = 70001
    lo, hi = v.reshape(-1, 3).min(0), v.reshape(-1, 3).max(0)
    o = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    k = rng.integers(0, len(v), n)
    aim = v[k].reshape(n, 3, 3).mean(1) - o
    d = np.where(rng.random(n)[:, None] < 0.5, aim, rng.normal(size=(n, 3))).astype(np.float32)
    if kind == "stack":
        d[::4] = (0.0, 0.0, -1.0)
    for ignore in (None, k.astype(np.int32)):
        got, want = s.trace_closest(o, d, ignore), s.trace_closest(o, d, ignore, width2=True)
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        tmax = np.where(np.isfinite(want[1]), want[1] * np.float32(1.000001), np.float32(1.0)).astype(np.float32)
        tmax[::3] = want[1][::3]
        assert np.array_equal(s.trace_any(o, d, tmax, ignore), s.trace_any(o, d, tmax, ignore, width2=True))
