"""Photon-mapped frames lit by each kind of light, whose direct light takes 1, 9 or 12 visibility
rays a hit: canvases of the small ones are kept in tests/golden/photon_lights.npz."""
import photon_scenes
import rednoise_b200 as rn

SPOT = dict(type=2, position=(0.1, 0.8, 0.3), direction=(-0.1, -1.0, -0.2), intensity=1.5, cone_cos=0.7)
LIGHTS = {
    "directional": [dict(type=1, direction=(-0.2, -0.9, -0.4), intensity=0.5)],
    "spot": [SPOT],
    "disk": [dict(radius=0.15, intensity=1.5)],
    "volume": [dict(type=3, radius=0.15, intensity=1.5)],
    "rectangle": [dict(type=4, intensity=2.0)],
    "triangle": [dict(type=5, intensity=2.0)],
    "three": [dict(type=4, intensity=1.0), SPOT, dict(type=3, position=(-0.4, 0.2, 0.4), radius=0.2, intensity=0.2)],
}
SMALL = (52, 39)
CAMERA = dict(position=(0.02, 0.05, 0.9))  # inside the room: every pixel hits something


def lights(name):
    return [rn.Light.default(**kw) for kw in LIGHTS[name]]


def render(scene, name, width=SMALL[0], height=SMALL[1], photons=1500):
    return scene.render_photon_mapped(width, height, photons, lights=lights(name), focal_length=1.2, **CAMERA)


def small(name):
    return render(photon_scenes.scene("panes" if name == "three" else "box"), name)
