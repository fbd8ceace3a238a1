"""Timed workloads of the renderer: what a program that uses rednoise_b200 has it do.

listed() names the standing cases, draw(rng) gives one more case of the same ranges,
prepare() builds what a program holds before the call (a prepared scene, cameras,
rays, image gradients), run() is one pass through the public entry points.

Scenes. "box" is the 36-triangle Cornell room of rednoise_b200.scenes, "sphere" the
room with a displaced, material-mixed icosphere of 20 * 4^size triangles (size 8 is
the 1.31M-triangle scene of bench.py), "soup" the room with size random triangles.
Reference-semantics renderers get the scene at the reference's scale (a room of
half-width 1, so its default light hangs under the ceiling, and its default camera at
z = 4 looks in).

Kinds, each with what it stands for:
* rays           closest hit and occlusion of device-resident rays (picking, baking,
                 visibility queries of a host application), any number of rays
* reference      renderPathTraced, the drop-in renderer, canvas on the host
* raytraced      renderRaytraced, Whitted preview frames, canvas on the host
* photon         renderPhotonMapped, canvas on the host
* bidirectional  renderBidirectional, the reference's row streams or counter streams
* metropolis     renderMetropolis
* physical       the radiance path tracer, image on the host (host = True) or, through
                 the PyTorch binding, on the device
* gradient       the PyTorch binding forward and backward over one or several views:
                 images and d(albedo), d(emission)
"""
import ctypes
import math

import numpy as np
import torch

import rednoise_b200 as rn
from rednoise_b200 import _native, scenes, torch_ops

ROOM = 1.0 / scenes.HALF  # room scaled to half-width 1
KINDS = ("rays", "reference", "raytraced", "photon", "bidirectional", "metropolis", "physical", "gradient")


def listed():
    return [
        # a host application asks for a few thousand rays at a time (one bundle of an
        # interactive tool): launch and call overhead count
        {"name": "rays-4k-box", "kind": "rays", "scene": "box", "size": 0, "rays": 4096},
        # a baking pass over a large scene: incoherent rays in one call
        {"name": "rays-2m-sphere8", "kind": "rays", "scene": "sphere", "size": 8, "rays": 2000003},
        # the drop-in's everyday call: the Cornell box at 320 x 240 and 16 samples
        {"name": "reference-320x240", "kind": "reference", "scene": "box", "size": 0, "width": 320, "height": 240,
         "spp": 16, "lights": 0, "aperture": 0.0},
        # the drop-in at full HD on the 1.31M-triangle scene
        {"name": "reference-1080p-sphere8", "kind": "reference", "scene": "sphere", "size": 8, "width": 1920,
         "height": 1080, "spp": 2, "lights": 0, "aperture": 0.0},
        # a Whitted frame of the same scene
        {"name": "raytraced-1080p-sphere8", "kind": "raytraced", "scene": "sphere", "size": 8, "width": 1920,
         "height": 1080, "shading": 2, "fog": 0.0},
        # photon mapping with the reference's default photon count
        {"name": "photon-200k-sphere7", "kind": "photon", "scene": "sphere", "size": 7, "width": 1280, "height": 720,
         "photons": 200000},
        # the reference's bidirectional renderer at its own image size, its own streams
        {"name": "bidirectional-640x480", "kind": "bidirectional", "scene": "box", "size": 0, "width": 640,
         "height": 480, "spp": 16, "rng": "reference"},
        # Metropolis with the reference's default number of mutations
        {"name": "metropolis-4m", "kind": "metropolis", "scene": "box", "size": 0, "width": 640, "height": 480,
         "mutations": 4000000},
        # the radiance path tracer on a small scene, as in the README
        {"name": "physical-720p-box", "kind": "physical", "scene": "box", "size": 0, "width": 1280, "height": 720,
         "spp": 64, "depth": 8, "rr": 3, "env": 0.0, "host": True},
        # and on the 1.31M-triangle scene at full HD, image kept on the device
        {"name": "physical-1080p-sphere8", "kind": "physical", "scene": "sphere", "size": 8, "width": 1920,
         "height": 1080, "spp": 32, "depth": 8, "rr": 3, "env": 0.0, "host": False},
        # inverse rendering of many materials: one view of the large scene
        {"name": "gradient-512-sphere8", "kind": "gradient", "scene": "sphere", "size": 8, "views": 1, "width": 512,
         "height": 512, "spp": 32, "depth": 6},
        # multi-view inverse rendering of a small scene
        {"name": "gradient-4x384-box", "kind": "gradient", "scene": "box", "size": 0, "views": 4, "width": 384,
         "height": 384, "spp": 16, "depth": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, lo, hi):
    """Width and height of an image of lo to hi pixels, aspect 1:1 to 16:9, odd sizes among them."""
    px, aspect = math.exp(rng.uniform(math.log(lo), math.log(hi))), rng.uniform(1.0, 16.0 / 9.0)
    return max(16, int(math.sqrt(px * aspect))), max(16, int(math.sqrt(px / aspect)))


def draw(rng):
    kind = rng.choice(KINDS)
    c = {"kind": kind, "scene": rng.choice(("box", "sphere", "sphere", "soup")), "size": 0}
    if kind in ("bidirectional", "metropolis"):
        c["scene"] = rng.choice(("box", "box", "sphere"))
    if c["scene"] == "sphere":
        c["size"] = rng.randint(3, 8)
    elif c["scene"] == "soup":
        c["size"] = _log_int(rng, 1e3, 2e5)
    dense = 8 if c["scene"] == "soup" else 1  # a random soup costs several times more per ray
    if kind == "rays":
        c["rays"] = _log_int(rng, 257, 2e6 / dense)
        return c
    w, h = _image(rng, 64 * 64, 1920 * 1080)
    if kind in ("bidirectional", "metropolis"):
        w, h = _image(rng, 96 * 96, 640 * 480)
    if kind == "gradient":
        w, h = _image(rng, 96 * 96, 512 * 512)
    c.update(width=w, height=h)
    px = w * h
    if kind == "reference":
        c.update(spp=max(1, min(_log_int(rng, 1, 64), 4000000 // dense // px)), lights=rng.choice((0, 0, 1, 2)),
                 aperture=rng.choice((0.0, 0.0, 0.05)))
    elif kind == "raytraced":
        c.update(shading=rng.randint(0, 2), fog=rng.choice((0.0, 0.08)))
    elif kind == "photon":
        c.update(photons=_log_int(rng, 5000, 200000))
        if c["scene"] == "soup":
            c["photons"] //= 4
    elif kind == "bidirectional":
        c.update(spp=_log_int(rng, 2, 16), rng=rng.choice(("reference", "reference", "counter")))
        if c["scene"] == "sphere":
            c["spp"] = max(1, c["spp"] // 4)
    elif kind == "metropolis":
        c.update(mutations=_log_int(rng, 50000, 4e6))
        if c["scene"] == "sphere":
            c["mutations"] //= 4
    elif kind == "physical":
        c.update(spp=max(1, min(_log_int(rng, 1, 64), 50000000 // dense // px)), depth=rng.randint(3, 10),
                 rr=rng.choice((3, 5, 64)), env=rng.choice((0.0, 0.0, 0.5)), host=rng.random() < 0.5)
    else:
        views = rng.randint(1, 4)
        c.update(views=views, spp=max(1, min(_log_int(rng, 4, 32), 8000000 // dense // (px * views))),
                 depth=rng.randint(3, 8))
    return c


# ---- scenes ------------------------------------------------------------------------


def _icosphere(level):
    tris = torch.from_numpy(np.ascontiguousarray(scenes.icosphere(0))).cuda()
    for _ in range(level):
        a, b, c = tris.unbind(1)
        ab, bc, ca = (torch.nn.functional.normalize(p + q, dim=1) for p, q in ((a, b), (b, c), (c, a)))
        tris = torch.stack([torch.stack(t, 1) for t in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))],
                           1).reshape(-1, 3, 3)
    return tris


def _added(case, rng):
    """The triangles that join the room: (vertices (n, 9), material (n,))."""
    if case["scene"] == "sphere":
        tris = _icosphere(case["size"])
        # radius 1.2 with seeded bumps of about 0.08, below the room's centre
        k = torch.from_numpy(rng.normal(size=(24, 3)) * rng.uniform(2.0, 14.0, (24, 1))).cuda()
        phase = torch.from_numpy(rng.uniform(0.0, 2.0 * math.pi, 24)).cuda()
        r = 1.2 + 0.02 * torch.sin(tris @ k.T + phase).sum(2, keepdim=True)
        v = (tris * r + torch.tensor([0.0, -1.45, 0.0], dtype=torch.float64, device="cuda")).float().cpu().numpy()
        u = rng.random(v.shape[0])
        return v.reshape(-1, 9), np.where(u < 0.6, 0, np.where(u < 0.85, 1, 2)).astype(np.int32)
    n = case["size"]
    c = rng.uniform(-scenes.HALF + 0.2, scenes.HALF - 0.2, (n, 3))
    d = rng.normal(size=(2, n, 3))
    d *= rng.uniform(0.01, 0.2, (2, n, 1)) / np.linalg.norm(d, axis=2, keepdims=True)
    return np.concatenate([c, c + d[0], c + d[1]], 1).astype(np.float32), np.zeros(n, np.int32)


def _scene(case, rng, scale=1.0):
    """(Scene, albedo, emission): the case's geometry with seeded materials, prepared."""
    # a light of ten times the quad's sides keeps the images' noise low, as in the tests
    room = scenes.cornell_box(light_scale=10.0)
    v, em = room["vertices"], room["emission"]
    mat = np.zeros(len(v), np.int32)
    if case["scene"] != "box":
        av, am = _added(case, rng)
        v, mat = np.concatenate([v, av]), np.concatenate([mat, am])
        em = np.concatenate([em, np.zeros((len(av), 3), np.float32)])
    n = len(v)
    em = em * np.float32(rng.uniform(0.8, 1.2))
    alb = rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32)
    par = np.where(mat == scenes.GGX, rng.uniform(0.05, 0.5, n), np.where(mat == scenes.DIELECTRIC, 1.5, 0.2))
    ref_mat = np.array([scenes.REF_DIFFUSE, scenes.REF_METAL, scenes.REF_GLASS], np.int32)[mat]
    ref_mat[em.max(1) > 0] = scenes.REF_EMISSIVE
    s = rn.Scene.from_arrays(np.ascontiguousarray(v * np.float32(scale)), albedo=alb, emission=em, material=mat,
                             material_param=par.astype(np.float32), ref_rgb=(alb * 255.0).astype(np.int32),
                             ref_material=ref_mat)
    s.prepare()
    return s, alb, em


def _views(case, rng):
    """Cameras near the standing one (in front of the room's open side), moved a little by the seed."""
    c = scenes.camera(case["width"], case["height"])
    out = []
    for _ in range(case.get("views", 1)):
        x, y, z = rng.uniform(-0.4, 0.4, 3)
        out.append(rn.Camera.make((x, y, c["position"][2] + z), c["target"], c["up"], c["vfov_deg"], case["width"],
                                  case["height"]))
    return out


def _lights(n, rng):
    out = []
    if n >= 1:  # a soft rectangle under the ceiling
        out.append(rn.Light.default(type=4, position=(0.0, 0.95, 0.0), intensity=float(rng.uniform(30, 50))))
    if n >= 2:  # a spot from the open side
        out.append(rn.Light.default(type=2, position=(0.3, 0.6, 1.5), direction=(-0.2, -0.4, -0.9), intensity=20.0,
                                 cone_cos=0.8))
    return out or None


def _ray_inputs(case, rng):
    n = case["rays"]
    o = rng.uniform(-scenes.HALF + 0.05, scenes.HALF - 0.05, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    # occlusion towards points of the ceiling light
    p = np.stack([rng.uniform(-0.6, 0.6, n), np.full(n, scenes.HALF - 2e-3), rng.uniform(-0.5, 0.5, n)], 1)
    to = p - o
    dist = np.linalg.norm(to, axis=1)
    return o, d, (to / dist[:, None]).astype(np.float32), (dist * 0.999).astype(np.float32)


# ---- the cases --------------------------------------------------------------------------


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"case": case}
    reference_scale = kind in ("reference", "raytraced", "photon", "bidirectional", "metropolis")
    st["scene"], alb, em = _scene(case, rng, ROOM if reference_scale else 1.0)
    if kind == "rays":
        st["rays"] = [torch.from_numpy(a).cuda() for a in _ray_inputs(case, rng)]
        return st
    if reference_scale:
        x, y = rng.uniform(-0.1, 0.1, 2)
        # the framing of the default call at 240 lines (focal length 2, the room's opening fills
        # five sixths of the height), whatever the image's height
        st["camera"] = dict(position=(float(x), float(y), 4.0), focal_length=2.0 * case["height"] / 240.0)
        st["lights"] = _lights(case.get("lights", 0), rng)
        st["seed"] = int(rng.integers(1 << 30))
        return st
    st["cameras"] = _views(case, rng)
    st["settings"] = rn.Settings.make(spp=case["spp"], max_depth=case["depth"], rr_depth=case.get("rr", case["depth"]),
                                      seed=int(rng.integers(1 << 30)), env=(case.get("env", 0.0),) * 3)
    if kind == "gradient" or not case["host"]:
        st["albedo"], st["emission"] = torch.from_numpy(alb).cuda(), torch.from_numpy(em).cuda()
        # the wavefront's frames are captured graphs: they need a stream other than the default one
        st["stream"] = torch.cuda.Stream()
    if kind == "gradient":
        st["albedo"].requires_grad_(True)
        st["emission"].requires_grad_(True)
        shape = (case["height"], case["width"], 3)
        st["d_images"] = [torch.from_numpy(rng.normal(size=shape).astype(np.float32)).cuda() for _ in st["cameras"]]
    return st


def _trace(scene, rays):
    lib = _native.load()
    o, d, sd, tmax = rays
    n = o.shape[0]
    tri, occ = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    t, u, v = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or 1)
    p = [ctypes.c_void_p(x.data_ptr()) for x in (o, d, sd, tmax, tri, t, u, v, occ)]
    flags = _native.RN_PT_DEVICE_POINTERS
    _native.check(lib.rn_pt_trace_closest(scene.handle, n, p[0], p[1], None, flags, stream, p[4], p[5], p[6], p[7]),
                  "trace_closest")
    _native.check(lib.rn_pt_trace_any(scene.handle, n, p[0], p[2], p[3], None, flags, stream, p[8]), "trace_any")
    return [tri, t, u, v, occ]


def _on_stream(stream, fn, st):
    """fn(st) on the program's own stream, joined with the current one before and after."""
    current = torch.cuda.current_stream()
    stream.wait_stream(current)
    with torch.cuda.stream(stream):
        out = fn(st)
    current.wait_stream(stream)
    return out


def _images(st):
    with torch.no_grad():
        return torch_ops.render(st["albedo"], st["emission"], st["scene"], [(st["cameras"][0], st["settings"])])


def _images_and_gradients(st):
    images = torch_ops.render(st["albedo"], st["emission"], st["scene"], [(c, st["settings"]) for c in st["cameras"]])
    grads = torch.autograd.grad(images, [st["albedo"], st["emission"]], st["d_images"])
    return [[i.detach() for i in images], list(grads)]


def run(st):
    case, scene = st["case"], st["scene"]
    kind = case["kind"]
    if kind == "rays":
        return _trace(scene, st["rays"])
    if kind == "physical":
        if case["host"]:
            return scene.render_physical(st["cameras"][0], st["settings"])
        return _on_stream(st["stream"], _images, st)
    if kind == "gradient":
        return _on_stream(st["stream"], _images_and_gradients, st)
    w, h, cam = case["width"], case["height"], st["camera"]
    if kind == "reference":
        return scene.render_reference(w, h, case["spp"], lights=st["lights"], aperture=case["aperture"], **cam)
    if kind == "raytraced":
        return scene.render_raytraced(w, h, shading=case["shading"], fog_density=case["fog"], **cam)
    if kind == "photon":
        return list(scene.render_photon_mapped(w, h, case["photons"], return_count=True, **cam))
    if kind == "bidirectional":
        return list(scene.render_bidirectional(w, h, case["spp"], rng=case["rng"], seed=st["seed"], want_rgb=True,
                                               **cam))
    return list(scene.render_metropolis(w, h, case["mutations"], seed=st["seed"], want_rgb=True, **cam))


def _triangles(case):
    return 36 + (20 * 4 ** case["size"] if case["scene"] == "sphere" else case["size"])


def work(case):
    """Bytes: the scene's triangles once (36 B of vertices, 32 B of shading where the pass
    shades), inputs and outputs. Flops: a ray needs at least the log2(n / 4) box tests on the
    way to one leaf (21 operations each) and that leaf's four triangle tests (60 each);
    rays per sample are counted at the estimator's lower end."""
    kind, n = case["kind"], _triangles(case)
    per_ray = 21.0 * max(1.0, math.log2(n / 4.0)) + 240.0
    if kind == "rays":
        return {"bytes": 36 * n + case["rays"] * (24 + 16 + 16 + 4), "flops": 2 * case["rays"] * per_ray}
    px = case["width"] * case["height"]
    if kind == "metropolis":
        return {"bytes": 68 * n + px * 16, "flops": case["mutations"] * 6 * per_ray}
    if kind == "photon":
        return {"bytes": 68 * n + px * 4 + case["photons"] * 48, "flops": (px * 10 + case["photons"] * 2) * per_ray}
    if kind == "raytraced":
        return {"bytes": 68 * n + px * 4, "flops": px * 10 * per_ray}
    if kind == "bidirectional":
        return {"bytes": 68 * n + px * 16, "flops": px * case["spp"] * 12 * per_ray}
    if kind == "reference":
        return {"bytes": 68 * n + px * 4, "flops": px * case["spp"] * 12 * per_ray}
    samples = px * case["spp"] * case.get("views", 1)
    if kind == "physical":
        return {"bytes": 84 * n + px * 12, "flops": samples * 4 * per_ray}
    return {"bytes": 108 * n + px * 24 * case["views"], "flops": samples * 8 * per_ray}


def exact(case, seed):
    """Distances of the closest hits by solving every ray against every triangle in 64 bits,
    where that is quick (which triangle it is, and so its barycentrics, has no single value:
    the room's boxes stand in the floor's plane). The renderers' canvases are whole numbers; the
    radiance and gradient images are Monte-Carlo sums whose every sample branches on rounded
    values (hit or miss, roulette, material choice), so they have no other value to be held
    against than the same samples'."""
    if case["kind"] != "rays" or case["rays"] * _triangles(case) > 1 << 28:
        return None
    rng = np.random.default_rng(seed)
    room = scenes.cornell_box(light_scale=10.0)
    v = room["vertices"]
    if case["scene"] != "box":
        v = np.concatenate([v, _added(case, rng)[0]])
    n = len(v)
    # the draws that _scene makes between the geometry and the rays
    rng.uniform(0.8, 1.2), rng.uniform(0.2, 0.8, (n, 3)), rng.uniform(0.05, 0.5, n)
    o, d, _, _ = (torch.from_numpy(a).double().cuda() for a in _ray_inputs(case, rng))
    tv = torch.from_numpy(v).double().cuda().reshape(-1, 3, 3)
    v0, e0, e1 = tv[:, 0], tv[:, 1] - tv[:, 0], tv[:, 2] - tv[:, 0]
    t_out = torch.full((len(o),), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // n)
    for i in range(0, len(o), step):
        oo, dd = o[i:i + step, None], d[i:i + step, None]
        p = torch.linalg.cross(dd, e1[None].expand(len(oo), -1, -1), dim=2)
        det = (e0 * p).sum(2)
        s = oo - v0
        a = (s * p).sum(2) / det
        q = torch.linalg.cross(s, e0[None].expand(len(oo), -1, -1), dim=2)
        b = (dd * q).sum(2) / det
        t = (e1 * q).sum(2) / det
        ok = (det.abs() >= 1e-8) & (a >= 0) & (b >= 0) & (a + b <= 1) & (t > 1e-5)
        t = torch.where(ok, t, math.inf)
        t_out[i:i + step] = t.amin(1)
    return [None, t_out, None, None, None]
