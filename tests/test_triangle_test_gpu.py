"""The paired triangle test against the reference's expressions in numpy float32, for the early-exit
form (ordinary launches, the 2-wide tree) and the straight form (launches of many rays)."""
import numpy as np
import pytest

import rednoise_b200 as rn

pytestmark = pytest.mark.gpu

f = np.float32


def reference_test(v, o, d):
    """t, u, v, det of rays against triangles, one by one, in the reference's order of float32 operations."""
    e0, e1, sp = v[:, 3:6] - v[:, 0:3], v[:, 6:9] - v[:, 0:3], o - v[:, 0:3]
    m0, m1, m2 = (-d).T, e0.T, e1.T
    det = m0[0] * (m1[1] * m2[2] - m2[1] * m1[2]) - m1[0] * (m0[1] * m2[2] - m2[1] * m0[2]) \
        + m2[0] * (m0[1] * m1[2] - m1[1] * m0[2])
    k = f(1.0) / det
    i00, i01, i02 = (m1[1] * m2[2] - m2[1] * m1[2]) * k, -(m0[1] * m2[2] - m2[1] * m0[2]) * k, \
        (m0[1] * m1[2] - m1[1] * m0[2]) * k
    i10, i11, i12 = -(m1[0] * m2[2] - m2[0] * m1[2]) * k, (m0[0] * m2[2] - m2[0] * m0[2]) * k, \
        -(m0[0] * m1[2] - m1[0] * m0[2]) * k
    i20, i21, i22 = (m1[0] * m2[1] - m2[0] * m1[1]) * k, -(m0[0] * m2[1] - m2[0] * m0[1]) * k, \
        (m0[0] * m1[1] - m1[0] * m0[1]) * k
    x, y, z = sp.T
    return i00 * x + i10 * y + i20 * z, i01 * x + i11 * y + i21 * z, i02 * x + i12 * y + i22 * z, det


@pytest.mark.parametrize("n,width2", [(4097, False), (4097, True), (131073, False)])
def test_hits_carry_the_reference_bits(n, width2):
    rng = np.random.default_rng(n)
    v = (rng.uniform(-1.0, 1.0, (300, 1, 3)) + rng.uniform(-0.3, 0.3, (300, 3, 3))).reshape(-1, 9).astype(f)
    v[:20, 3:6] = v[:20, 0:3] + f(1e-3) * (v[:20, 6:9] - v[:20, 0:3]) + f(1e-5)  # slivers
    s = rn.Scene.from_arrays(v)
    o = rng.uniform(-1.5, 1.5, (n, 3)).astype(f)
    target = np.einsum("ij,ijk->ik", rng.dirichlet((1, 1, 1), n), v[rng.integers(0, len(v), n)].reshape(-1, 3, 3))
    d = (target - o).astype(f)
    idx, t, u, w = s.trace_closest(o, d, width2=width2)[:4]
    hit = idx >= 0
    assert hit.mean() > 0.9
    want = reference_test(v[idx[hit]], o[hit], d[hit])
    for got, ref in zip((t, u, w), want):
        assert np.array_equal(got[hit].view(np.uint32), ref.view(np.uint32))
    # what was missed has no hit well inside a triangle (the reference rejects |det| < 1e-8)
    for i in np.flatnonzero(~hit)[:64]:
        tt, uu, ww, det = reference_test(v, np.broadcast_to(o[i], (len(v), 3)), np.broadcast_to(d[i], (len(v), 3)))
        assert not ((tt > 1e-4) & (uu > 1e-3) & (ww > 1e-3) & (uu + ww < 0.999) & (np.abs(det) >= 1e-8)).any()
