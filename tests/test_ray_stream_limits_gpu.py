"""Closest-hit queries around the numbers of rays and triangles from which lanes take the next ray
when theirs is done, against the 2-wide reference tree."""
import numpy as np
import pytest

import rednoise_b200 as rn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris,n", [(767, 262144), (768, 262143), (768, 262144), (769, 262145),
                                    (1500, 148 * 7 * 4 * 32 * 2 + 17)])
def test_queries_equal_the_reference_tree(tris, n):
    rng = np.random.default_rng(tris + n)
    size = 1.3 ** (np.arange(tris) % 60)[:, None, None]  # rays of very different lengths
    v = rng.uniform(-1.0, 1.0, (tris, 1, 3)) * size + size * rng.uniform(-1.0, 1.0, (tris, 3, 3))
    v = np.ascontiguousarray(v.reshape(-1, 9), np.float32)
    s = rn.Scene.from_arrays(v)
    o = rng.uniform(v.reshape(-1, 3).min(0), v.reshape(-1, 3).max(0), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[::997] = (0.0, 1.0, 0.0)  # rays for the 2-wide tree among the others
    d[5::1009] = np.nan
    k = rng.integers(0, tris, n).astype(np.int32)
    for ignore in (None, k):
        got, want = s.trace_closest(o, d, ignore), s.trace_closest(o, d, ignore, width2=True)
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
