"""What a program that uses this framework has it do, as cases to be timed.

Each case goes through the public entry points alone: ray batches
(Trace.trace_rays_device, Trace.occluded_device), sampling passes of a tracer
(Trace.sample, Trace.sample_adaptive, with and without a radiance cache) and
the denoiser (Denoiser.denoise_device).  The scenes are the procedural ones of
pfx_b200.synth at the sizes of the benchmark, the clip and the tests.  A tracer
runs with the launch choices it is created with.

A scene's description and packed buffers are kept between preparations, as a
program keeps the scene it renders; the tracer, the camera, the sample seeds,
the rays and the images are made anew from the seed each time.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from pfx_b200 import synth
from pfx_b200.cache import CacheSettings, RadianceCache
from pfx_b200.denoise import Denoiser, write_tza
from pfx_b200.trace import Adaptive, SceneBuffers, Settings, Trace


def listed():
    return [
        # Picking and probe queries of a tool: a few thousand closest-hit rays
        # of finite reach into a small scene, where the latency of one call counts.
        {"name": "rays_probe", "kind": "rays", "scene": "spheres", "triangles": 20000, "any": False, "rays": 4097,
         "reach": 100.0},
        # A host that drives its own integrator: closest hits of a large batch
        # of camera rays and rays scattered from their hits, in the 1.19 M
        # triangle room.
        {"name": "rays_closest_room", "kind": "rays", "scene": "room", "triangles": 1200000, "any": False,
         "rays": 1 << 21, "reach": 1e20},
        # The same host's shadow rays towards the room's 128 lights.
        {"name": "rays_shadow_room", "kind": "rays", "scene": "room", "triangles": 1200000, "any": True,
         "rays": 1500001, "reach": 1e20},
        # Looking about while setting up a shot: one sample of a small window
        # after every camera move, the pcg sampler.
        {"name": "preview_320", "kind": "still", "scene": "room", "triangles": 100000, "width": 320, "height": 180,
         "spp": 1, "sampler": "pcg", "moves": True, "aperture": 0.0},
        # The small still of the benchmark: 512 x 512, 16 samples, depth 4,
        # three rectangle lights.
        {"name": "still_512", "kind": "still", "scene": "spheres", "triangles": 20000, "width": 512, "height": 512,
         "spp": 16, "sampler": "sobol", "moves": True, "aperture": 0.0},
        # One frame of the clip: 1280 x 720, 16 samples, 100k triangles and 128
        # lights, the camera moved before every frame.
        {"name": "clip_720p", "kind": "still", "scene": "room", "triangles": 100000, "width": 1280, "height": 720,
         "spp": 16, "sampler": "sobol", "moves": True, "aperture": 0.0},
        # A film of odd size through a lens with an aperture, refined two
        # samples at a time with the pcg sampler.
        {"name": "lens_1919x1081", "kind": "still", "scene": "room", "triangles": 400000, "width": 1919,
         "height": 1081, "spp": 2, "sampler": "pcg", "moves": False, "aperture": 0.1},
        # Adaptive render to 64 samples of the instanced scene (200k instanced
        # triangles, 128 lights): rounds over ever fewer pixels.
        {"name": "adaptive_instanced", "kind": "adaptive", "scene": "instances", "triangles": 200000, "width": 960,
         "height": 540, "spp": 64, "sampler": "sobol", "moves": True, "aperture": 0.0},
        # The headline benchmark's step: one sample of every pixel of the 4K
        # room, accumulating.
        {"name": "room_4k", "kind": "still", "scene": "room", "triangles": 1200000, "width": 3840, "height": 2160,
         "spp": 1, "sampler": "sobol", "moves": False, "aperture": 0.0},
        # A 1080p frame of the same room refined with the radiance cache, which
        # the passes before have trained and this one trains on: inference and
        # training in the pass.
        {"name": "room_1080p_cached", "kind": "cached", "scene": "room", "triangles": 1200000, "width": 1920,
         "height": 1080, "spp": 1, "sampler": "sobol", "moves": False, "aperture": 0.0},
        # The finished 4K frame denoised from its films on the device (two tiles).
        {"name": "denoise_4k", "kind": "denoise", "width": 3840, "height": 2160},
        # A small image of ragged size denoised while it is worked on.
        {"name": "denoise_517x391", "kind": "denoise", "width": 517, "height": 391},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["rays", "rays", "still", "still", "adaptive", "denoise"])
    if kind == "denoise":
        return {"kind": kind, "width": int(_log(rng, 96, 3840)), "height": int(_log(rng, 96, 2160))}
    scene = rng.choice(["room", "room", "spheres", "instances"])
    triangles = {"room": int(_log(rng, 10000, 1200000)), "spheres": 20000,
                 "instances": int(_log(rng, 20000, 200000))}[scene]
    case = {"kind": kind, "scene": scene, "triangles": triangles}
    if kind == "rays":
        case.update({"any": rng.random() < 0.5, "rays": int(_log(rng, 1000, 1 << 21)), "reach": 1e20})
        return case
    width = int(_log(rng, 160, 1920 if kind == "still" else 640))
    height = max(90, int(width * rng.uniform(0.5, 0.75)))
    spp = int(_log(rng, 16, 64.99)) if kind == "adaptive" else int(_log(rng, 1, 16.99))
    if kind == "still":  # a drawn case costs no more than the largest listed one
        spp = max(1, min(spp, 8000000 // (width * height)))
    case.update({"width": width, "height": height, "spp": spp, "sampler": rng.choice(["sobol", "sobol", "pcg"]),
                 "moves": rng.random() < 0.5, "aperture": rng.choice([0.0, 0.0, 0.05])})
    return case


# ------------------------------------------------------------------ scenes
_scenes: dict = {}


def _scene(case):
    """(scene, settings, packed buffers) of a case, kept between preparations."""
    sampler = case.get("sampler", "sobol")
    key = (case["scene"], case["triangles"], sampler)
    if key not in _scenes:
        while len(_scenes) >= 6:
            _scenes.pop(next(iter(_scenes)))
        if case["scene"] == "spheres":
            w = synth.plain_512(sampler=sampler)
        elif case["scene"] == "instances":
            w = synth.instanced_1080(target=case["triangles"], sampler=sampler)
        else:
            w = synth.room_4k(target=case["triangles"], meshes_n=max(1, round(case["triangles"] / 4000)),
                              sampler=sampler)
        _scenes[key] = (w.scene, w.settings, SceneBuffers(w.scene, w.settings))
    return _scenes[key]


def _camera(case, rng, aspect):
    """A camera of the scene's usual standpoint, moved and turned a little."""
    if case["scene"] == "spheres":
        eye, target, fov = (0, 9, 34), (0, 8, 0), 45.0
    elif case["scene"] == "instances":
        eye, target, fov = (0, 35, 130), (0, 15, 0), 50.0
    else:
        eye, target, fov = (0, 5, 14.0), (0, 4, 0), 60.0
    eye = np.asarray(eye, float) + rng.uniform(-0.5, 0.5, 3)
    target = np.asarray(target, float) + rng.uniform(-1.0, 1.0, 3)
    return synth.look_at(tuple(eye), tuple(target), fov, aspect)


# ------------------------------------------------------------------ states
def _prepare_rays(case, seed):
    scene, settings, buffers = _scene(case)
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    trace = Trace(scene, settings, 64, 36, buffers=buffers)
    n = case["rays"]
    uniform = lambda *shape: torch.rand(shape, generator=g, device="cuda")  # noqa: E731

    def batch(o, d, limit):
        out = torch.zeros((len(d), 8), device="cuda")
        out[:, 0:3], out[:, 3], out[:, 4:7] = o, limit, d
        return out

    def hits_of(rays):
        hits = torch.empty((len(rays), 4), dtype=torch.int32, device="cuda")
        trace.trace_rays_device(rays.data_ptr(), len(rays), hits.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return hits

    # camera rays of a 3840 x 2160 frame in scanline order from a random
    # pixel on, for two thirds of the batch; the rest leave their hits again,
    # into the half space that the camera ray came from
    cam = _camera(case, rng, 16 / 9)
    first = n if case["any"] else max(1, (2 * n) // 3)
    pixel = (int(rng.integers(0, 3840 * 2160)) + torch.arange(first, device="cuda")) % (3840 * 2160)
    x = ((pixel % 3840) + uniform(first)) / 3840 * 2 - 1
    y = (torch.div(pixel, 3840, rounding_mode="floor") + uniform(first)) / 2160 * 2 - 1
    axis = lambda v: torch.tensor(np.asarray(v, np.float32), device="cuda")  # noqa: E731
    d = axis(cam.forward) + axis(cam.right) * x[:, None] - axis(cam.up) * y[:, None]
    d = torch.nn.functional.normalize(d, dim=1)
    eye = axis(cam.origin).expand(first, 3)
    rays = batch(eye, d, case["reach"])
    hits = hits_of(rays)
    t = torch.where(hits[:, 3] == 1, hits[:, 0].view(torch.float32), torch.full_like(d[:, 0], 20.0))
    point = eye + d * (t - 1e-3 * t.clamp(min=1.0))[:, None]
    if case["any"]:
        if len(scene.lights):
            lights = axis(scene.lights["position"])
            aim = lights[torch.randint(0, len(lights), (n,), generator=g, device="cuda")]
        else:
            aim = point + 10 * torch.randn((n, 3), generator=g, device="cuda")
        to = aim - point
        distance = to.norm(dim=1).clamp(min=1e-6)
        rays = batch(point, to / distance[:, None], distance * 0.9999 - 0.0002)
        out = torch.empty(n, dtype=torch.int32, device="cuda")
    else:
        more = n - first
        if more:
            away = torch.nn.functional.normalize(
                torch.nn.functional.normalize(torch.randn((more, 3), generator=g, device="cuda"), dim=1) - d[:more],
                dim=1)
            rays = torch.cat([rays, batch(point[:more], away, case["reach"])])
        out = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    return {"case": case, "trace": trace, "rays": rays.contiguous(), "out": out}


def _prepare_trace(case, seed):
    scene, settings, buffers = _scene(case)
    rng = np.random.default_rng(seed)
    camera = _camera(case, rng, case["width"] / case["height"])
    trace = Trace(dataclasses.replace(scene, camera=camera), settings, case["width"], case["height"], buffers=buffers)
    if case["aperture"] > 0.0:
        trace.set_lens(aperture=case["aperture"], focus_distance=10.0)
    state = {"case": case, "trace": trace, "camera": camera, "seed": int(rng.integers(0, 1 << 30)),
             "films": trace.films_device()}
    for film in state["films"]:
        film.owner = trace  # the films are the tracer's own memory: whoever holds them holds the tracer
    if case["kind"] == "cached":
        state["cache"] = RadianceCache(CacheSettings(seed=int(rng.integers(0, 1 << 30))))
        trace.set_cache(state["cache"])
        for _ in range(96):  # the passes before this one have trained the cache
            trace.sample(1, state["seed"])
    return state


_LAYERS = [("enc_conv0", 32, 9), ("enc_conv1", 32, 32), ("enc_conv2", 48, 32), ("enc_conv3", 64, 48),
           ("enc_conv4", 80, 64), ("enc_conv5a", 96, 80), ("enc_conv5b", 96, 96), ("dec_conv4a", 112, 160),
           ("dec_conv4b", 112, 112), ("dec_conv3a", 96, 160), ("dec_conv3b", 96, 96), ("dec_conv2a", 64, 128),
           ("dec_conv2b", 64, 64), ("dec_conv1a", 64, 73), ("dec_conv1b", 32, 64), ("dec_conv0", 3, 32)]


def _weights():
    """Weights of the filter's shapes: random, exact in FP16, and scaled so that
    the images that come out have the range of the images that go in."""
    rng = np.random.default_rng(11)
    w = {}
    for name, out, inputs in _LAYERS:
        gain = 0.05 if name == "dec_conv0" else 1.0
        w[name + ".weight"] = (gain * rng.normal(0, np.sqrt(2.0 / (9 * inputs)), (out, inputs, 3, 3))).astype(np.float16)
        w[name + ".bias"] = rng.uniform(0.2, 0.3, out).astype(np.float16) if name == "dec_conv0" else \
            rng.normal(0, 0.02, out).astype(np.float16)
    return w


def _images(case, seed):
    """Noisy colour with a high range, albedo and normals of a frame (RGBA32F)."""
    h, w = case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    smooth = lambda c: torch.nn.functional.interpolate(  # noqa: E731
        torch.rand((1, c, max(2, h // 40), max(2, w // 40)), generator=g, device="cuda"), (h, w), mode="bilinear")[0]
    colour, albedo, normal = (torch.ones((h, w, 4), device="cuda") for _ in range(3))
    light = torch.exp(4.0 * smooth(3) - 3.0 + 0.6 * torch.randn((3, h, w), generator=g, device="cuda"))
    albedo[..., :3] = smooth(3).permute(1, 2, 0)
    colour[..., :3] = light.permute(1, 2, 0) * albedo[..., :3]
    normal[..., :3] = torch.nn.functional.normalize(2.0 * smooth(3) - 1.0, dim=0).permute(1, 2, 0)
    return colour, albedo, normal


def _prepare_denoise(case, seed):
    return {"case": case, "denoiser": Denoiser(write_tza(_weights())), "images": _images(case, seed),
            "out": torch.empty((case["height"], case["width"], 4), device="cuda")}


def prepare(case, seed):
    if case["kind"] == "rays":
        return _prepare_rays(case, seed)
    if case["kind"] == "denoise":
        return _prepare_denoise(case, seed)
    return _prepare_trace(case, seed)


def run(state):
    case = state["case"]
    if case["kind"] == "rays":
        rays, out, stream = state["rays"], state["out"], torch.cuda.current_stream().cuda_stream
        if case["any"]:
            state["trace"].occluded_device(rays.data_ptr(), len(rays), out.data_ptr(), stream)
            return out
        state["trace"].trace_rays_device(rays.data_ptr(), len(rays), out.data_ptr(), stream)
        return {"t": out[:, 0].view(torch.float32), "ids": out[:, 1:]}
    if case["kind"] == "denoise":
        c, a, n = state["images"]
        state["denoiser"].denoise_device(case["width"], case["height"], c.data_ptr(), a.data_ptr(), n.data_ptr(),
                                         state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["out"]
    trace = state["trace"]
    if case["moves"]:
        trace.set_camera(state["camera"])
    if case["kind"] == "adaptive":
        done = trace.sample_adaptive(Adaptive(threshold=0.01, min_samples=8, max_samples=case["spp"], growth=1.5),
                                     state["seed"])
        return {"films": state["films"], "rounds": [[r.samples, r.active] for r in done.rounds]}
    trace.sample(case["spp"], state["seed"])
    return state["films"]


# ------------------------------------------------------------------ work
def work(case):
    """The bytes that a pass reads and writes once, and the operations of the
    tests it cannot avoid: per ray two box tests (24 operations) a level of a
    binary tree over the triangles and two triangle tests (46); per path of a
    sampling pass six such rays; per convolution its multiply-adds."""
    if case["kind"] == "denoise":
        pixels = case["width"] * case["height"]
        level = {"enc_conv2": 1, "dec_conv2": 1, "enc_conv3": 2, "dec_conv3": 2, "enc_conv4": 3, "dec_conv4": 3,
                 "enc_conv5": 4}
        macs = sum(9 * o * i * pixels / 4 ** level.get(name[:9], 0) for name, o, i in _LAYERS)
        return {"bytes": 64 * pixels, "flops": 2 * macs}
    ray = 2 * 24 * math.log2(case["triangles"]) + 2 * 46
    scene = 150 * case["triangles"]
    if case["kind"] == "rays":
        return {"bytes": case["rays"] * (36 if case["any"] else 48) + scene, "flops": case["rays"] * ray}
    pixels = case["width"] * case["height"]
    spp = case["spp"] if case["kind"] != "adaptive" else 0.6 * case["spp"]
    paths = pixels * spp
    # accumulation read and written, three films written
    return {"bytes": pixels * (96 + 48) + scene, "flops": paths * 6 * ray}


# ------------------------------------------------------------------ exact values
def _exact_rays(case, seed):
    """Closest hits of the small scene by testing every triangle in 64 bits."""
    state = _prepare_rays(case, seed)
    scene, _, _ = _scene(case)
    v = torch.tensor(np.asarray(scene.triangles["v"], np.float32).reshape(-1, 3, 3), device="cuda").double()
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = []
    for rays in state["rays"].double().split(64):
        o, d, limit = rays[:, None, 0:3], rays[:, None, 4:7], rays[:, 3]
        pv = torch.linalg.cross(d.expand(-1, len(a), 3), e2.expand(len(rays), -1, 3))
        det = (e1 * pv).sum(2)
        inv = 1.0 / torch.where(det.abs() < 1e-9, torch.ones_like(det), det)
        sv = o - a
        u = (sv * pv).sum(2) * inv
        qv = torch.linalg.cross(sv, e1.expand(len(rays), -1, 3))
        w = (d * qv).sum(2) * inv
        t = (e2 * qv).sum(2) * inv
        miss = (det.abs() < 1e-9) | (u < 0) | (u > 1) | (w < 0) | (u + w > 1) | (t <= 1e-4) | (t >= limit[:, None])
        out.append(torch.minimum(torch.where(miss, torch.full_like(t, math.inf), t).min(1).values, limit))
    return {"t": torch.cat(out), "ids": None}


def _exact_denoise(case, seed):
    """The filter in 64 bits: exposure, transfer function, U-Net, and back."""
    colour, albedo, normal = (x.double()[..., :3] for x in _images(case, seed))
    h, w = case["height"], case["width"]
    # exposure: 0.18 over the geometric mean of the mean luminance of bins of about 16 x 16 pixels
    gy, gx = -(-h // 16), -(-w // 16)
    lum = colour.clamp(min=0.0) @ torch.tensor([0.212671, 0.715160, 0.072169], dtype=torch.float64, device="cuda")
    ys = torch.tensor([j * h // gy for j in range(gy + 1)], device="cuda")
    xs = torch.tensor([i * w // gx for i in range(gx + 1)], device="cuda")
    total = torch.nn.functional.pad(lum.cumsum(0).cumsum(1), (1, 0, 1, 0))[ys][:, xs]
    sums = total[1:, 1:] - total[:-1, 1:] - total[1:, :-1] + total[:-1, :-1]
    mean = sums / (ys.diff()[:, None] * xs.diff()[None, :])
    kept = mean[mean > 1e-8]
    scale = 0.18 / 2.0 ** kept.log2().mean() if len(kept) else torch.tensor(1.0, dtype=torch.float64, device="cuda")
    top = 1.92653250e-1 * math.log(65504.0 + 6.260261e-3) + 9.9862015e-1
    y = (colour * scale).clamp(min=0.0)
    y = torch.where(y <= 1.57945760e-06, 1.41283765e+03 * y,
                    torch.where(y <= 3.22087631e-02, 1.64593172e+00 * y ** 4.31384981e-01 - 2.94139609e-03,
                                1.92653254e-01 * torch.log(y + 6.26026094e-03) + 9.98620152e-01)) / top
    x = torch.cat([y, albedo.clamp(0.0, 1.0), normal.clamp(-1.0, 1.0) * 0.5 + 0.5], dim=2).permute(2, 0, 1)[None]
    # sides rounded up to 16, the image in the corner of zeros
    x = torch.nn.functional.pad(x, (0, -w % 16, 0, -h % 16))
    weights = {k: torch.tensor(v.astype(np.float64), device="cuda") for k, v in _weights().items()}
    conv = lambda name, v: torch.relu(torch.nn.functional.conv2d(  # noqa: E731
        v, weights[name + ".weight"], weights[name + ".bias"], padding=1))
    pool = lambda v: torch.nn.functional.max_pool2d(v, 2)  # noqa: E731
    up = lambda v, skip: torch.cat([torch.nn.functional.interpolate(v, scale_factor=2), skip], 1)  # noqa: E731
    p1 = pool(conv("enc_conv1", conv("enc_conv0", x)))
    p2 = pool(conv("enc_conv2", p1))
    p3 = pool(conv("enc_conv3", p2))
    v = pool(conv("enc_conv4", p3))
    v = conv("enc_conv5b", conv("enc_conv5a", v))
    v = conv("dec_conv4b", conv("dec_conv4a", up(v, p3)))
    v = conv("dec_conv3b", conv("dec_conv3a", up(v, p2)))
    v = conv("dec_conv2b", conv("dec_conv2a", up(v, p1)))
    v = conv("dec_conv0", conv("dec_conv1b", conv("dec_conv1a", up(v, x))))
    v = v[0, :, :h, :w].permute(1, 2, 0) * top
    v = torch.where(v <= 2.23151711e-03, v / 1.41283765e+03,
                    torch.where(v <= 3.70974749e-01,
                                ((v + 2.94139609e-03) / 1.64593172e+00).clamp(min=0.0) ** (1.0 / 4.31384981e-01),
                                torch.exp((v - 9.98620152e-01) / 1.92653254e-01) - 6.26026094e-03)) / scale
    return torch.cat([v, torch.ones_like(v[..., :1])], dim=2)


def exact(case, seed):
    if case["kind"] == "rays" and not case["any"] and case["rays"] <= 8192 and case["scene"] == "spheres":
        return _exact_rays(case, seed)
    if case["kind"] == "denoise" and -(-case["width"] // 16) * -(-case["height"] // 16) * 256 <= 1 << 20:
        return _exact_denoise(case, seed)
    return None  # a path's estimate follows the sampler's sequence: no value but the tracer's own
