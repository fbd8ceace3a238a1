"""Many closest-hit queries (lanes that take the next ray when theirs is done) against the 2-wide
reference tree, either side of the number of rays from which they run and with remainders."""
import numpy as np
import pytest

import rednoise_b200 as rn
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [131071, 131072, 131073, 148 * 7 * 4 * 32 * 2 + 17])
@pytest.mark.parametrize("kind", ["room", "chain"])
def test_many_rays_equal_the_reference_tree(kind, n):
    rng = np.random.default_rng(n)
    if kind == "room":
        v = scenes.icosphere_scene(4)["vertices"]
    else:  # sizes that grow by halves: rays of very different lengths
        size = 1.4 ** (np.arange(900) % 90)[:, None, None]
        v = (rng.uniform(-1.0, 1.0, (900, 1, 3)) * size + size * rng.uniform(-1.0, 1.0, (900, 3, 3)))
    v = np.ascontiguousarray(v.reshape(-1, 9), np.float32)
    s = rn.Scene.from_arrays(v)
    o = rng.uniform(v.reshape(-1, 3).min(0), v.reshape(-1, 3).max(0), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[::997] = (0.0, 1.0, 0.0)  # rays for the 2-wide tree among the others
    d[5::1009] = np.nan
    k = rng.integers(0, len(v), n).astype(np.int32)
    for ignore in (None, k):
        got, want = s.trace_closest(o, d, ignore), s.trace_closest(o, d, ignore, width2=True)
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
