"""Metropolis at the numbers of chains where the launch changes: the estimate does not depend on how
chains are laid out over threads, so b and the image's mean follow the bootstrap alone."""
import numpy as np
import pytest

import rednoise_b200 as rn
from rednoise_b200 import scenes

pytestmark = pytest.mark.gpu

ROOM = 148 * 2 * 128


@pytest.mark.parametrize("chains", [1, 33, 2368, 2369, ROOM // 2, ROOM // 2 + 1, ROOM, ROOM + 1])
def test_every_chain_deposits_its_steps(chains):
    v = scenes.cornell_box()["vertices"] * np.float32(1.0 / 8.0)
    s = rn.Scene.from_arrays(v)
    steps = 3
    argb, rgb, b = s.render_metropolis(48, 40, mutations=chains * steps, chains=chains, bootstrap=4096, seed=5,
                                       want_rgb=True)
    assert b > 0.0
    # each mutation deposits weights that sum to 1 in luminance, scaled to b on average
    lum = rgb.astype(np.float64) @ np.array([0.2126, 0.7152, 0.0722])
    assert abs(lum.mean() / b - 1.0) < 1e-3
