"""Small photon-mapped frames whose canvases are kept in tests/golden/photon_canvases.npz:
one photon, frames that are not whole pixel tiles, photons that take more draws than
the first table of stream positions holds, and pixels with many diffuse hits behind glass."""
import numpy as np

import rednoise_b200 as rn
from rednoise_b200 import scenes

SCALE = np.float32(1.0 / scenes.HALF)
# name: (scene, width, height, photons, gather rays)
FRAMES = {
    "one_photon": ("box", 17, 9, 1, 0),
    "odd_frame": ("box", 61, 45, 3001, 0),
    "long_draws": ("white", 40, 24, 2000, 0),
    "mixed": ("sphere", 64, 48, 5000, 0),
    "behind_glass": ("panes", 50, 41, 2500, 0),
    "final_gather": ("box", 9, 5, 1500, 3),
}


def _quad(z, s=1.2):
    a, b, c, d = (-s, -s, z), (s, -s, z), (s, s, z), (-s, s, z)
    return [np.array(t, np.float32).reshape(9) for t in ((a, b, c), (a, c, d))]


def scene(kind):
    sc = scenes.icosphere_scene(3) if kind == "sphere" else scenes.cornell_box(light_scale=10.0)
    v, rgb, mat = sc["vertices"] * SCALE, sc["ref_rgb"].copy(), sc["ref_material"].copy()
    if kind == "white":
        rgb[mat == scenes.REF_DIFFUSE] = 255
    if kind == "panes":  # three panes of glass between the camera and the room
        panes = np.stack([t for z in (1.2, 1.5, 1.8) for t in _quad(z)])
        v = np.concatenate([v, panes])
        rgb = np.concatenate([rgb, np.full((6, 3), 255, np.int32)])
        mat = np.concatenate([mat, np.full(6, scenes.REF_GLASS, np.int32)])
    return rn.Scene.from_arrays(np.ascontiguousarray(v), ref_rgb=rgb, ref_material=mat)


def render(name):
    """(canvas, stored photons) of one frame."""
    kind, w, h, photons, gather = FRAMES[name]
    return scene(kind).render_photon_mapped(w, h, photons, gather_rays=gather, position=(0.05, 0.1, 4.0),
                                            focal_length=2.0 * h / 240.0, return_count=True)
