"""The workloads this renderer is timed on, as a program that uses it calls them.

Every case goes through the package's public entry points: Camera.render
(host frame), mypbr_gpu_render_device (frame stays on the GPU, caller's
stream), render_batch, denoise and display. Scenes are the package's own
generators: the Cornell box, the sphere field under an HDRI, the triangle room
and the voxel hall.

A state's inputs come from its seed: the random stream of the render, the
camera, and for the small scenes (Cornell box, sphere field) the scene handle
and its contents too. The two large scenes are loaded once per size and
rendered from many cameras, as the frames of an animation are.

A render's per-path estimates are random numbers; no value in 64 bits exists
for them, so exact() answers for the denoiser and the display path only.
"""
import collections
import ctypes
import math
import random
import tempfile

import numpy as np
import torch

import mypbr_gb300 as mp
from mypbr_gb300 import workloads

DEVICE = "cuda:0"


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # The smallest call: one pass of a viewer's thumbnail while the user turns the camera.
        _render("cornell_preview_64_1spp", "cornell", 64, 64, 1, depth=8, entry="host"),
        # The Cornell box at its stock settings: many bounces, few paths.
        _render("cornell_256_64spp", "cornell", 256, 256, 64, depth=50, entry="host"),
        # The headline workload (1000 spheres under an HDRI), a quarter of its samples.
        _render("spheres_1080p_64spp", "spheres", 1920, 1080, 64, depth=16, entry="device"),
        # An odd-sized frame for the denoiser (albedo, normal, variance) through haze, clear glass letting light by.
        _render("spheres_haze_guides_853x479_24spp", "spheres", 853, 479, 24, depth=16, entry="host", haze=True,
                features=True, transparent=True),
        # 2 million triangles, 32 principled materials, 16 lamps: a tree larger than the L2 cache.
        _render("room_2m_1080p_16spp", "room", 1920, 1080, 16, depth=12, entry="device", size=2_000_000),
        # The 512^3 voxel world under the atmosphere sky, plain.
        _render("hall_512_960x540_32spp", "hall", 960, 540, 32, depth=16, entry="device", size=512),
        # The same world with the guiding network at work: a frame after training has ended.
        _render("hall_512_guided_640x360_48spp", "hall", 640, 360, 48, depth=16, entry="device", size=512,
                guided=8),
        # The start of a guided render of a new frame: recorded waves and the network's first training steps.
        _render("hall_512_training_480x270_64spp", "hall", 480, 270, 64, depth=16, entry="device", size=512,
                guided=8, training=True),
        # A band of rows of a larger frame, one worker's share of a frame split over several.
        _render("room_300k_band_1280x720_32spp", "room", 1280, 720, 32, depth=12, entry="device", size=300_000,
                band=True),
        # Uneven small scenes with denoiser guides in one call, half of them hazy.
        {"name": "batch_12_scenes", "kind": "batch", "jobs": 12, "largest": 512, "spp": 96},
        # The denoiser on a frame that is on the GPU already.
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080},
        # Bloom, vignette and tone mapping of a host frame into display bytes.
        {"name": "display_1080p", "kind": "display", "width": 1920, "height": 1080, "tonemap": "aces", "bloom": 0.1,
         "vignette": 0.3},
    ]


def _render(name, scene, width, height, spp, depth, entry, size=0, haze=False, features=False, transparent=False,
            guided=0, training=False, band=False):
    case = {"kind": "render", "scene": scene, "width": width, "height": height, "spp": spp, "depth": depth,
            "entry": entry, "size": size, "haze": haze, "features": features, "transparent": transparent,
            "guided": guided, "training": training, "band": band}
    if name:
        case["name"] = name
    return case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame(rng, lo, hi):
    """A width and height of lo to hi pixels in all, any aspect between 1:1 and 2:1, even and odd sizes."""
    pixels = _log_int(rng, lo, hi)
    width = max(16, int(math.sqrt(pixels * rng.uniform(1.0, 2.0))))
    return width, max(16, pixels // width)


def draw(rng):
    kind = rng.choice(["cornell", "cornell", "spheres", "spheres", "room", "room", "hall", "hall", "guided",
                       "training", "batch", "denoise", "display"])
    entry = rng.choice(["host", "device"])
    if kind == "batch":
        return {"kind": "batch", "jobs": rng.randint(2, 12), "largest": _log_int(rng, 96, 512),
                "spp": _log_int(rng, 4, 96)}
    if kind == "denoise":
        width, height = _frame(rng, 64 * 64, 1920 * 1080)
        return {"kind": "denoise", "width": width, "height": height}
    if kind == "display":
        width, height = _frame(rng, 64 * 64, 1920 * 1080)
        return {"kind": "display", "width": width, "height": height,
                "tonemap": rng.choice(["none", "reinhard", "aces"]), "bloom": rng.choice([0.0, 0.1]),
                "vignette": rng.choice([0.0, 0.3])}
    features, band = rng.random() < 0.3, entry == "device" and rng.random() < 0.25
    if kind == "cornell":
        width, height = _frame(rng, 64 * 64, 640 * 640)
        spp = max(1, min(_log_int(rng, 1, 256), 24_000_000 // (width * height)))
        return _render("", "cornell", width, height, spp, rng.choice([8, 16, 50]), entry,
                       haze=rng.random() < 0.4, features=features, band=band)
    if kind == "spheres":
        width, height = _frame(rng, 64 * 64, 1920 * 1080)
        spp = max(1, min(_log_int(rng, 1, 128), 100_000_000 // (width * height)))
        haze = rng.random() < 0.4
        if haze:
            spp = max(1, min(spp, 24_000_000 // (width * height)))
        return _render("", "spheres", width, height, spp, 16, entry, haze=haze, features=features,
                       transparent=rng.random() < 0.4, band=band)
    if kind == "room":
        width, height = _frame(rng, 64 * 64, 1920 * 1080)
        spp = max(1, min(_log_int(rng, 1, 64), 20_000_000 // (width * height)))
        return _render("", "room", width, height, spp, 12, entry, size=rng.choice([10_000, 60_000, 300_000]),
                       features=features, band=band)
    size = rng.choice([128, 256])
    if kind == "hall":
        width, height = _frame(rng, 64 * 64, 1280 * 720)
        spp = max(1, min(_log_int(rng, 1, 64), 20_000_000 // (width * height)))
        return _render("", "hall", width, height, spp, 16, entry, size=size, features=features, band=band)
    hidden = rng.choice([2, 4, 8])
    if kind == "guided":
        width, height = _frame(rng, 64 * 64, 640 * 360)
        spp = max(1, min(_log_int(rng, 4, 64), 10_000_000 // (width * height)))
        return _render("", "hall", width, height, spp, 16, "device", size=size, guided=hidden)
    # training: at most four recorded waves, before the mixture is first sampled
    width, height = _frame(rng, 128 * 128, 480 * 270)
    spp = max(1, min(_log_int(rng, 4, 64), 8_000_000 // (width * height)))
    return _render("", "hall", width, height, spp, 16, "device", size=size, guided=hidden, training=True)


# ------------------------------------------------------------------ scenes

_hosts = collections.OrderedDict()  # the large scenes by size, and the handles made from them
_loaded = collections.OrderedDict()
_HAZE = "material haze volume 0.9 0.9 0.9 g 0.6\nfog 0.02 haze\n"


def _write_scene(directory, scene, seed, size=0, haze=False):
    if scene == "cornell":
        path = workloads.cornell_scene(directory)
    elif scene == "spheres":
        path = workloads.sphere_field_scene(directory, seed=seed)
    elif scene == "room":
        path = workloads.triangle_room_scene(directory, triangles=size)
    else:
        path = workloads.voxel_hall_scene(directory, size=size)
    if haze:
        with open(path, "a") as f:
            f.write(_HAZE)
    return path


def _load(scene, seed, size=0, haze=False):
    with tempfile.TemporaryDirectory() as directory:
        return mp.load_scene(_write_scene(directory, scene, seed, size, haze))


def _kept(store, key, make, most):
    if key not in store:
        store[key] = make()
    store.move_to_end(key)
    while len(store) > most:
        store.popitem(last=False)
    return store[key]


def _scene(case, seed):
    """(host scene, GPU handle) of a case; the large ones are kept, a few of them."""
    if case["scene"] in ("cornell", "spheres"):
        host = _load(case["scene"], seed, haze=case["haze"])
        return host, mp.GpuScene(host)
    host = _kept(_hosts, (case["scene"], case["size"]), lambda: _load(case["scene"], 0, case["size"]), 4)

    def handle():
        gpu = mp.GpuScene(host)
        if case["guided"]:  # the network is made by the handle's first guided render, from that render's seed
            cam = mp.Camera(*host.camera.structs())
            cam.image_width, cam.samples_per_pixel, cam.seed, cam.guided = 16, 1, 1, case["guided"]
            cam.render(gpu)
            mp.guide_reset(gpu)
            if not case["training"]:
                # sampled from the first wave on and trained no further
                mp.guide_schedule(gpu, max_steps=0, use_after=0)
        return gpu

    # a network belongs to its handle: a guided case has one of its own
    return host, _kept(_loaded, (case["scene"], case["size"], case["guided"], case["training"]), handle, 6)


def _aim(cam, scene, size, rng):
    """Moves the camera of a generated scene a little, as the next frame of an animation does."""
    if scene == "cornell":
        cam.lookfrom = (278 + rng.uniform(-60, 60), 278 + rng.uniform(-60, 60), -800 + rng.uniform(-20, 40))
    elif scene == "spheres":
        a = rng.uniform(0, 2 * math.pi)
        cam.lookfrom = (18 * math.sin(a), 6 + rng.uniform(-1, 1), 18 * math.cos(a))
    elif scene == "room":
        cam.lookfrom = (rng.uniform(-0.1, 0.1), 3.2 + rng.uniform(-0.5, 0.5), -13.5)
        cam.lookat = (rng.uniform(-2, 2), 2.6 + rng.uniform(-0.5, 0.5), 0)
    else:
        s = size / 512.0
        cam.lookfrom = ((-90 + rng.uniform(-3, 3)) * s, (130 + rng.uniform(-3, 3)) * s,
                        (-60 + rng.uniform(-3, 3)) * s)
        cam.lookat = ((60 + rng.uniform(-10, 10)) * s, 120 * s, (10 + rng.uniform(-10, 10)) * s)


def _camera(host, case, rng):
    cam = mp.Camera(*host.camera.structs())
    cam.image_width = case["width"]
    cam.aspect_ratio = case["width"] / (case["height"] + 0.5)  # height() rounds down to the case's
    cam.samples_per_pixel = case["spp"]
    cam.max_depth = case["depth"]
    cam.seed = rng.getrandbits(48)
    cam.collect_features = case["features"]
    cam.transparent_shadows = case["transparent"]
    cam.guided = case["guided"]
    if case["band"]:
        cam.first_row = case["height"] // 3
        cam.row_count = case["height"] // 3 + 1
    _aim(cam, case["scene"], case["size"], rng)
    return cam


def _planes(height, width, features):
    """Radiance, albedo, normal and variance buffers on the GPU (the last three for guides only)."""
    out = [torch.zeros(height, width, 3, dtype=torch.float64, device=DEVICE)]
    if features:
        out += [torch.zeros_like(out[0]), torch.zeros_like(out[0]),
                torch.zeros(height, width, dtype=torch.float64, device=DEVICE)]
    return out


# ------------------------------------------------------------------ prepare

def prepare(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "render":
        host, gpu = _scene(case, seed)
        cam = _camera(host, case, rng)
        state = {"kind": "render", "entry": case["entry"], "cam": cam, "gpu": gpu, "host": host,
                 "training": case["training"]}
        if case["entry"] == "device":
            state["planes"] = _planes(cam.height(), case["width"], case["features"])
            state["stream"] = torch.cuda.Stream(DEVICE)
        return state
    if case["kind"] == "batch":
        jobs, keep = [], []
        for k in range(case["jobs"]):
            scene = ("room", "cornell", "spheres")[k % 3]
            width = max(32, int(case["largest"] * (1.0 - 0.75 * k / case["jobs"])))
            sub = _render("", scene, width, width, max(1, case["spp"] // (1 + k % 4)), 12, "device",
                          size=10_000 if scene == "room" else 0, haze=k % 2 == 1, features=True)
            if scene == "room":
                host = _load("room", 0, sub["size"], sub["haze"])
            else:
                host = _load(scene, seed + k, haze=sub["haze"])
            gpu, cam = mp.GpuScene(host), _camera(host, sub, rng)
            planes = _planes(cam.height(), width, True)
            keep.append((host, gpu, planes))
            jobs.append((gpu, cam, *(p.data_ptr() for p in planes)))
        return {"kind": "batch", "jobs": jobs, "keep": keep}
    if case["kind"] == "denoise":
        rad, alb, nrm, var = _noisy_frame(case, seed)
        return {"kind": "denoise", "frame": (rad, alb, nrm, var), "out": torch.empty_like(rad)}
    return {"kind": "display", "frame": _hdr_frame(case, seed),
            "opts": mp.display_opts(exposure=0.5, tonemap=case["tonemap"], bloom=case["bloom"],
                                    vignette=case["vignette"])}


def _noisy_frame(case, seed):
    """A low-sample render as the denoiser meets it: flat and textured regions, edges in albedo and
    normal, noise of the stated variance, one pixel in 500 a firefly."""
    g = torch.Generator(DEVICE)
    g.manual_seed(seed)
    h, w = case["height"], case["width"]

    def uniform(*shape):
        return torch.rand(*shape, generator=g, device=DEVICE, dtype=torch.float64)

    y, x = torch.meshgrid(torch.arange(h, device=DEVICE), torch.arange(w, device=DEVICE), indexing="ij")
    region = (x * 9 // w) * 7 + y * 7 // h
    alb = 0.1 + 0.8 * uniform(64, 3)[region % 64] * (0.8 + 0.2 * uniform(h, w, 1))
    nrm = torch.nn.functional.normalize(uniform(64, 3)[(region // 2) % 64] - 0.5, dim=-1)
    light = 0.2 + 2.0 * uniform(64, 1)[(region // 3) % 64] + 0.5 * torch.sin(x / 40.0)[..., None] ** 2
    deviation = 0.3 * light[..., 0]
    rad = alb * light * (1.0 + 0.3 * torch.randn(h, w, 1, generator=g, device=DEVICE, dtype=torch.float64)).clamp_min(0)
    spark = uniform(h, w) < 0.002
    rad = torch.where(spark[..., None], rad * 40.0, rad)
    var = torch.where(spark, (40.0 * deviation) ** 2, deviation ** 2)
    return rad.contiguous(), alb.contiguous(), nrm.contiguous(), var.contiguous()


def _hdr_frame(case, seed):
    """A frame of high dynamic range on the host, as Camera.render returns it."""
    rng = np.random.default_rng(seed)
    frame = rng.lognormal(-1.0, 1.0, (case["height"], case["width"], 3))
    lamps = rng.random((case["height"], case["width"])) < 0.001
    frame[lamps] *= 50.0
    return frame


# ------------------------------------------------------------------ run

def run(state):
    if state["kind"] == "batch":
        mp.render_batch(state["jobs"])
        return [planes for _, _, planes in state["keep"]]
    if state["kind"] == "denoise":
        rad, alb, nrm, var = state["frame"]
        h, w = var.shape
        # denoise works on the legacy stream, which other tensors' work here shares
        mp.denoise(rad.data_ptr(), alb.data_ptr(), nrm.data_ptr(), var.data_ptr(), w, h, state["out"].data_ptr(),
                   on_device=True)
        return state["out"]
    if state["kind"] == "display":
        return mp.display(state["frame"], state["opts"])
    if state["training"]:
        mp.guide_reset(state["gpu"])  # a new frame: a fresh network
    if state["entry"] == "host":
        frame = state["cam"].render(state["gpu"])
        return [frame.radiance, frame.albedo, frame.normal, frame.variance]
    c, o = state["cam"].structs()
    planes = [ctypes.c_void_p(p.data_ptr()) for p in state["planes"]] + [None] * (4 - len(state["planes"]))
    mp.check(mp.lib().mypbr_gpu_render_device(state["gpu"].handle, ctypes.byref(c), ctypes.byref(o), *planes,
                                              ctypes.c_void_p(state["stream"].cuda_stream), None))
    return state["planes"]


# ------------------------------------------------------------------ work

# Per scene: rays (extension and shadow) a path casts on average, as mypbr_render_stats counts them on the
# listed cases, and estimates of the interior nodes such a ray has to visit and of its primitive tests.
_RAYS = {"cornell": (6.0, 5, 3), "spheres": (3.6, 14, 3), "room": (5.9, 40, 6), "hall": (6.2, 30, 8)}
_NODE_FLOPS, _PRIM_FLOPS, _SHADE_FLOPS = 24, 40, 300


def _render_work(scene, pixels, spp, features, size, guided, depth):
    rays, nodes, prims = _RAYS[scene]
    flops = pixels * spp * rays * (nodes * _NODE_FLOPS + prims * _PRIM_FLOPS + _SHADE_FLOPS)
    if guided:  # the network at up to four vertices of a path
        flops += pixels * spp * 4 * 2 * (128 * 64 + guided * 64 * 64)
    # the frame written once; the scene read once
    scene_bytes = {"cornell": 4e3, "spheres": 1024 * 512 * 28 + 1e5, "room": 112.0 * size, "hall": 1.2 * size ** 3 / 4}
    return pixels * 8 * (10 if features else 3) + scene_bytes[scene], flops


def work(case):
    if case["kind"] == "render":
        rows = case["height"] // 3 + 1 if case["band"] else case["height"]
        b, f = _render_work(case["scene"], case["width"] * rows, case["spp"], case["features"], case["size"],
                            case["guided"], case["depth"])
        return {"bytes": b, "flops": f}
    if case["kind"] == "batch":
        total_b = total_f = 0.0
        for k in range(case["jobs"]):
            scene = ("room", "cornell", "spheres")[k % 3]
            width = max(32, int(case["largest"] * (1.0 - 0.75 * k / case["jobs"])))
            b, f = _render_work(scene, width * width, max(1, case["spp"] // (1 + k % 4)), True, 10_000, 0, 12)
            total_b, total_f = total_b + b, total_f + f
        return {"bytes": total_b, "flops": total_f}
    n = case["width"] * case["height"]
    if case["kind"] == "denoise":
        return {"bytes": n * 8 * 13, "flops": n * (5 * (25 * 26 + 20) + 60)}
    bloom = 1.34 * 22 * 6 / 4 + 60 if case["bloom"] > 0 else 0
    return {"bytes": n * (24 + 24 + 3), "flops": n * (100 + bloom)}


# ------------------------------------------------------------------ exact

def exact(case, seed):
    if case["kind"] == "denoise":
        return _exact_denoise(*_noisy_frame(case, seed))
    if case["kind"] == "display":
        frame = torch.from_numpy(_hdr_frame(case, seed)).to(DEVICE)
        return (_exact_postprocess(frame, case["bloom"], case["vignette"]).cpu().numpy(), None)
    return None


def _luminance(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _shifted(img, dy, dx, fill=0.0):
    """img at (y + dy, x + dx), `fill` outside."""
    out = torch.full_like(img, fill)
    h, w = img.shape[:2]
    y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = img[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _exact_denoise(rad, alb, nrm, var):
    """Firefly clamp, then five edge-avoiding a-trous iterations with a variance-guided luminance weight."""
    eps = 1e-3
    light = rad / (alb + eps)
    var = var / _luminance(alb + eps) ** 2
    # fireflies: an inner pixel above its eight neighbours with a deviation over half its luminance
    lum = _luminance(light)
    around = torch.zeros_like(lum)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            if dx or dy:
                around = torch.maximum(around, _shifted(lum, dy, dx))
    inner = torch.zeros_like(lum, dtype=torch.bool)
    inner[1:-1, 1:-1] = True
    clamp = inner & (lum > 0) & (var.sqrt() >= 0.5 * lum) & (lum > around)
    scale = torch.where(clamp, around / lum, torch.ones_like(lum))
    light, var = light * scale[..., None], var * scale ** 2
    inside = torch.ones_like(var)
    kern = (1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16)
    for it in range(5):
        step = 1 << it
        total, weight = torch.zeros_like(var), torch.zeros_like(var)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                c = (0.5, 0.25)[abs(dx)] * (0.5, 0.25)[abs(dy)]
                total += c * _shifted(var, dy, dx)
                weight += c * _shifted(inside, dy, dx)
        sigma = 4.0 * (total / weight).clamp_min(0).sqrt() + 1e-10
        lum = _luminance(light)
        acc, wsum, vsum = torch.zeros_like(light), torch.zeros_like(var), torch.zeros_like(var)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                sy, sx = dy * step, dx * step
                if abs(sy) >= var.shape[0] or abs(sx) >= var.shape[1]:
                    continue
                q = _shifted(light, sy, sx)
                e = ((nrm - _shifted(nrm, sy, sx)) ** 2).sum(-1) / 0.01 + \
                    ((alb - _shifted(alb, sy, sx)) ** 2).sum(-1) / 0.01 + (lum - _luminance(q)).abs() / sigma
                wgt = kern[dy + 2] * kern[dx + 2] * torch.exp(-e) * _shifted(inside, sy, sx)
                acc += wgt[..., None] * q
                wsum += wgt
                vsum += wgt * wgt * _shifted(var, sy, sx)
        light, var = acc / wsum[..., None], vsum / wsum ** 2
    return light * (alb + eps)


def _at(img, j, i):
    """img at rows j and columns i, edges repeated."""
    return img[j.clamp(0, img.shape[0] - 1)][:, i.clamp(0, img.shape[1] - 1)]


def _exact_postprocess(img, bloom, vignette, threshold=1.0, radius=0.04):
    """Bloom from a half-size pyramid of Gaussian-blurred bright parts, then vignetting."""
    h, w, _ = img.shape
    dev = img.device
    out = img.clone()
    if bloom > 0:
        lum = _luminance(img)
        keep = torch.isfinite(lum) & (lum > threshold)
        level = torch.where(keep[..., None], img * ((lum - threshold) / lum)[..., None], torch.zeros_like(img))
        taps = [math.exp(-0.5 * k * k / 2.25) for k in range(-5, 6)]
        glow, count = torch.zeros_like(img), 0
        for _ in range(min(max(math.ceil(math.log2(max(radius * w, 1.0))), 1), 10)):
            if level.shape[0] <= 1 or level.shape[1] <= 1:
                break
            lh, lw = max(1, level.shape[0] // 2), max(1, level.shape[1] // 2)
            j, i = torch.arange(lh, device=dev), torch.arange(lw, device=dev)
            level = 0.25 * (_at(level, 2 * j, 2 * i) + _at(level, 2 * j, 2 * i + 1) + _at(level, 2 * j + 1, 2 * i) +
                            _at(level, 2 * j + 1, 2 * i + 1))
            soft = sum(t / sum(taps) * _at(level, j, i + k - 5) for k, t in enumerate(taps))
            soft = sum(t / sum(taps) * _at(soft, j + k - 5, i) for k, t in enumerate(taps))
            y = (torch.arange(h, device=dev, dtype=torch.float64) + 0.5) * (lh / h) - 0.5
            x = (torch.arange(w, device=dev, dtype=torch.float64) + 0.5) * (lw / w) - 0.5
            jy, ix = y.floor().long(), x.floor().long()
            fy, fx = (y - jy)[:, None, None], (x - ix)[None, :, None]
            glow += (1 - fy) * ((1 - fx) * _at(soft, jy, ix) + fx * _at(soft, jy, ix + 1)) + \
                fy * ((1 - fx) * _at(soft, jy + 1, ix) + fx * _at(soft, jy + 1, ix + 1))
            count += 1
        if count:
            out = out + bloom / count * glow
    if vignette > 0:
        dy = torch.arange(h, device=dev, dtype=torch.float64)[:, None] + 0.5 - 0.5 * h
        dx = torch.arange(w, device=dev, dtype=torch.float64)[None, :] + 0.5 - 0.5 * w
        f = 1 + vignette * (dx * dx + dy * dy) / (0.25 * w * w + 0.25 * h * h)
        out = out / (f * f)[..., None]
    return out
