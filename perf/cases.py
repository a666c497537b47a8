"""Performance cases: what a user of this renderer has it do, through its public entry points.

A case is a dict of plain values: `kind` is the entry point, `scene` the scene family, the rest
are its sizes and options. The scenes are the repository's own workloads and example
configurations (mandelbulber_gb300/workloads.py, tests/golden): the power-8 Mandelbulb and the
scale-2 Mandelbox in front of the camera, a quaternion set with the finite-difference estimate,
a Menger sponge with lights and reflections, a camera a millionth from the surface.
A seed moves the camera around the object and draws the light, the palette and the points, so
that every seed is another frame of the same work.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import mandelbulber_gb300 as mb
from mandelbulber_gb300 import diff as D
from mandelbulber_gb300 import workloads as W

_context = None


def _ctx() -> mb.Context:
    """The one context that a user's program keeps."""
    global _context
    if _context is None:
        _context = mb.Context(0)
    return _context


def listed() -> list:
    return [
        # a preview window while the camera is being moved: the smallest call, its latency counts
        {"name": "preview_bulb_160x120", "kind": "still", "scene": "bulb", "w": 160, "h": 120, "prec": "fp32"},
        # the Mandelbulb still of the benchmark's first configuration
        {"name": "still_bulb_640x480", "kind": "still", "scene": "bulb", "w": 640, "h": 480, "prec": "fp32"},
        # the headline frame: Mandelbox with hard shadows, ray-traced AO, fog and glow at 1080p
        {"name": "still_box_1920x1080", "kind": "still", "scene": "box", "w": 1920, "h": 1080, "prec": "fp32"},
        # the command line's render: layers into host memory, an odd size near the default 800x600
        {"name": "host_box_801x601", "kind": "host", "scene": "box", "w": 801, "h": 601, "prec": "fp32"},
        # the reference's own arithmetic (FP64 policy), as for a final check of a frame
        {"name": "fp64_box_481x271", "kind": "still", "scene": "box", "w": 481, "h": 271, "prec": "fp64"},
        # a deep zoom, where the AUTO policy has to leave FP32
        {"name": "auto_deepzoom_192x192", "kind": "still", "scene": "deep", "w": 192, "h": 192, "prec": "auto"},
        # a quaternion set: finite-difference estimate, FP64 under every policy
        {"name": "delta_quaternion_320x240", "kind": "still", "scene": "delta", "w": 320, "h": 240, "prec": "fp32"},
        # secondary effects: predefined lights, fast AO and ray-traced reflections on a sponge
        {"name": "effects_menger_480x270", "kind": "still", "scene": "menger", "w": 480, "h": 270, "prec": "fp32"},
        # frames of a flight animation, mixed resolutions, in one call
        {"name": "flight_8_frames", "kind": "batch", "frames": 8, "downscale": 1},
        # a fitting step: gradients of eight frames by power, camera and light
        {"name": "grad_8x256", "kind": "grad", "frames": 8, "size": 256},
        # post-processing of a finished frame: 16-bit image and screen-space ambient occlusion
        {"name": "post_1920x1080_q20", "kind": "post", "w": 1920, "h": 1080, "quality": 20},
        # distance estimates at a point cloud (sampling a volume for a mesh)
        {"name": "distance_box_2m", "kind": "distance", "scene": "box", "n": 2000003, "prec": "fp64"},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["still", "still", "still", "host", "fp64", "deep", "delta", "menger", "batch", "grad", "post",
                       "distance"])
    aspect = rng.choice([4 / 3, 16 / 9, 1.0, 3 / 4, 2.37])

    def size(lo, hi):   # a frame of lo .. hi pixels, odd sizes among them
        n = _log(rng, lo, hi)
        w = max(32, int(math.sqrt(n * aspect)))
        return {"w": w, "h": max(32, min(n // w, hi // w))}

    if kind == "still":
        return {"kind": "still", "scene": rng.choice(["bulb", "box"]), "prec": "fp32", **size(64 * 48, 1920 * 1080)}
    if kind == "host":
        return {"kind": "host", "scene": rng.choice(["bulb", "box"]), "prec": "fp32", **size(96 * 54, 1280 * 720)}
    if kind == "fp64":
        return {"kind": "still", "scene": "box", "prec": "fp64", **size(64 * 48, 481 * 271)}
    if kind == "deep":
        return {"kind": "still", "scene": "deep", "prec": "auto", **size(48 * 48, 192 * 192)}
    if kind == "delta":
        return {"kind": "still", "scene": "delta", "prec": "fp32", **size(48 * 32, 320 * 240)}
    if kind == "menger":
        return {"kind": "still", "scene": "menger", "prec": "fp32", **size(64 * 48, 480 * 270)}
    if kind == "batch":
        return {"kind": "batch", "frames": rng.randint(2, 8), "downscale": rng.choice([1, 2, 3, 5])}
    if kind == "grad":
        return {"kind": "grad", "frames": rng.randint(1, 8), "size": _log(rng, 48, 256)}
    if kind == "post":
        return {"kind": "post", "quality": rng.randint(6, 20), **size(96 * 54, 1920 * 1080)}
    return {"kind": "distance", "scene": rng.choice(["bulb", "box"]), "n": _log(rng, 1000, 2000003),
            "prec": rng.choice(["fp32", "fp64"])}


_PREC = {"fp32": mb.PREC_FP32_FIX, "fp64": mb.PREC_FP64, "auto": mb.PREC_AUTO}
_LAYERS = {"image_float": (3, torch.float32), "zbuffer": (1, torch.float32), "alpha": (1, torch.int16),
           "opacity": (1, torch.int16), "colour": (3, torch.uint8)}


def _view(radius, seed) -> dict:
    """A seeded camera at `radius` from the origin that looks at it, light and palette."""
    rng = np.random.default_rng(seed)
    az, el = math.radians(rng.uniform(-12, 12)), math.radians(rng.uniform(-12, 12))
    pos = radius * np.array([math.sin(az) * math.cos(el), -math.cos(az) * math.cos(el), math.sin(el)])
    a, b = W.look_angles(-pos)
    return {"view_point_x": float(pos[0]), "view_point_y": float(pos[1]), "view_point_z": float(pos[2]),
            "angle_alfa": a, "angle_beta": b, "main_light_alfa": math.radians(rng.uniform(38, 52)),
            "main_light_beta": math.radians(rng.uniform(38, 52)), "coloring_random_seed": int(rng.integers(1, 999999))}


def _scene(case, seed):
    w, h, family = case["w"], case["h"], case["scene"]
    if family == "bulb":
        return W.workload("mandelbulb_640x480", w, h, **_view(3.5, seed))
    if family == "box":
        return W.workload("mandelbox_1080p", w, h, **_view(20.0, seed))
    if family == "deep":
        return W.make_scene({**W.MANDELBULB_640x480, "N": 1000, **_deep_view(w, h, seed)})
    if family == "delta":   # the settings of the "quaternion - lathe" example
        return W.workload("mandelbulb_640x480", w, h, **{**_view(3.0, seed), "formula": 5, "analityc_DE_mode": 0,
                                                         "DE_factor": 0.5, "penetrating_lights": 1,
                                                         "glow_intensity": 1})
    return W.workload("mandelbulb_640x480", w, h, **{
        **W.AUX_LIGHTS, **_view(3.6, seed), "formula": 7, "N": 50, "ambient_occlusion_enabled": 1,
        "fast_ambient_occlusion_mode": 1, "raytraced_reflections": 1, "reflections_max": 2, "reflect": 0.4,
        "glow_intensity": 1, "aux_light_predefined_1_enabled": 1, "aux_light_predefined_1_x": 3.0,
        "aux_light_predefined_1_y": -3.0, "aux_light_predefined_1_z": 3.0, "aux_light_predefined_1_intensity": 1.3,
        "aux_light_predefined_2_enabled": 1, "aux_light_predefined_2_x": -3.0, "aux_light_predefined_2_y": -3.0,
        "aux_light_predefined_2_z": 0.0, "aux_light_predefined_2_intensity": 3.0})


def _deep_view(w, h, seed) -> dict:
    """A camera 1e-6 in front of a surface point of the Mandelbulb, found by tracing a seeded
    ray with plain 64-bit arithmetic."""
    rng = np.random.default_rng(seed)
    origin = np.array([0.0, -3.5, 0.0])
    while True:
        d = np.array([0.0, 1.0, 0.0]) + rng.normal(0.0, 0.15, 3)
        d /= np.linalg.norm(d)
        t = 0.0
        for _ in range(20000):
            de = _bulb_scalar(origin + d * t, 1000)
            if de < 1e-12 or t > 10.0:
                break
            t += de
        if de < 1e-12:
            break
    footprint = 10.0 ** rng.uniform(-8.5, -7.5)
    cam = origin + d * (t - 1e-6)
    a, b = W.look_angles(d)
    return {"image_width": w, "image_height": h, "view_point_x": float(cam[0]), "view_point_y": float(cam[1]),
            "view_point_z": float(cam[2]), "angle_alfa": a, "angle_beta": b, "perspective": footprint * w / 1e-6}


def _bulb_scalar(p, N) -> float:
    x, y, z = (float(v) for v in p)
    cx, cy, cz, dr = x, y, z, 1.0
    r = math.sqrt(x * x + y * y + z * z)
    for _ in range(N):
        th, ph, r7 = 8.0 * math.asin(z / r), 8.0 * math.atan2(y, x), r ** 7
        dr = 8.0 * r7 * dr + 1.0
        q = r7 * r
        x, y, z = q * math.cos(th) * math.cos(ph) + cx, q * math.cos(th) * math.sin(ph) + cy, q * math.sin(th) + cz
        r = math.sqrt(x * x + y * y + z * z)
        if r > 100.0:
            return 0.5 * r * math.log(r) / dr
    return 0.0


def _buffers(w, h) -> dict:
    return {k: torch.zeros((h, w, c) if c > 1 else (h, w), dtype=t, device="cuda") for k, (c, t) in _LAYERS.items()}


def _pointers(buffers) -> dict:
    return {k: v.data_ptr() for k, v in buffers.items()}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ctx": _ctx()}
    if kind == "still":
        s["scene"], s["prec"] = _scene(case, seed), _PREC[case["prec"]]
        s["out"] = _buffers(case["w"], case["h"])
        s["layers"] = _pointers(s["out"])
    elif kind == "host":
        s["scene"], s["prec"] = _scene(case, seed), _PREC[case["prec"]]
        s["image"] = mb.CImage.empty(case["w"], case["h"])
    elif kind == "batch":
        frames = W.flight(n_keys=8, frames_per_key=4, seed=seed, downscale=case["downscale"])[:case["frames"]]
        # every resolution of the flight in turn, so that a seed changes the views and not the work
        for i, f in enumerate(frames):
            w, h = (v // case["downscale"] for v in W.FLIGHT_RESOLUTIONS[i % 4])
            for k, v in (("image_width", w), ("image_height", h), ("perspective", repr(W.fov_persp(w, h)))):
                mb.scene_set(f, k, v)
            # the spline may pass through the bulb; the camera stays in the keyframes' shell
            r = math.sqrt(sum(f.vp[k] ** 2 for k in range(3)))
            for k in range(3):
                f.vp[k] *= min(max(r, 2.0), 4.0) / r
            mb.finalize(f)
        s["scenes"] = frames
        s["out"] = [_buffers(f.image_width, f.image_height) for f in frames]
        s["layers"] = [_pointers(b) for b in s["out"]]
    elif kind == "grad":
        scenes, theta, _ = D.grad_batch(case["frames"], case["size"], seed)
        s["renderer"] = D.Renderer(s["ctx"], scenes)
        s["renderer"].set_theta(theta)
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["frames"], case["size"], case["size"], 3)
        s["dL"] = torch.randn(shape, generator=g, device="cuda")   # a loss's derivative by the images
        s["jacobian"] = torch.zeros(shape + (D.GRAD_PARAMS,), device="cuda")
    elif kind == "post":
        w, h = case["w"], case["h"]
        s["scene"] = W.workload("mandelbox_1080p", w, h, **_view(20.0, seed), post_SSAO_enabled=1,
                                post_SSAO_quality=case["quality"], ambient_occlusion_enabled=0)
        s["buffers"] = _buffers(w, h)
        s["ctx"].render_device(s["scene"], _pointers(s["buffers"]))
        s["image16"] = torch.zeros((h, w, 3), dtype=torch.int16, device="cuda")
        p = {k: ctypes.c_void_p(v.data_ptr()) for k, v in s["buffers"].items()}
        s["c_layers"] = mb.mbgb_image(w, h, p["image_float"], p["zbuffer"], p["alpha"], p["opacity"], p["colour"],
                                      None, None, None)
    else:
        n = case["n"]
        s["scene"] = W.workload("mandelbox_1080p" if case["scene"] == "box" else "mandelbulb_640x480", 640, 480)
        s["prec"] = _PREC[case["prec"]]
        s["points"], s["detail"] = _points(case, seed)
        s["out"] = {"distance": torch.zeros(n, dtype=torch.float64, device="cuda"),
                    "iterations": torch.zeros(n, dtype=torch.int32, device="cuda"),
                    "max_iter": torch.zeros(n, dtype=torch.uint8, device="cuda")}
    return s


def _points(case, seed):
    """Points of a cube around the object, as a volume sampling takes them, and detail sizes."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    half = 6.5 if case["scene"] == "box" else 1.3
    points = (torch.rand((case["n"], 3), generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * half
    detail = torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64) * 1e-3 * half + 1e-6
    return points, detail


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "still":
        ctx.render_device(s["scene"], s["layers"], precision=s["prec"])
        return s["out"]
    if kind == "host":
        im = ctx.render(s["scene"], s["image"], precision=s["prec"])
        return {"image_float": im.image_float, "zbuffer": im.zbuffer, "alpha": im.alpha, "opacity": im.opacity,
                "colour": im.colour, "hit": im.hit, "iters": im.iters, "depth": im.depth}
    if kind == "batch":
        ctx.render_batch_device(s["scenes"], s["layers"])
        return s["out"]
    if kind == "grad":
        r = s["renderer"]
        grad = r.backward(s["dL"], s["jacobian"])
        return {"dtheta": grad, "image": r.image, "jacobian": s["jacobian"]}
    if kind == "post":
        lib, sc = mb.library(), s["scene"]
        st = lib.mbgb_compile_image16_device(ctx._h, ctypes.byref(sc), s["buffers"]["image_float"].data_ptr(),
                                             sc.image_width, sc.image_height, s["image16"].data_ptr())
        st = st or lib.mbgb_ssao_device(ctx._h, ctypes.byref(sc), ctypes.byref(s["c_layers"]), s["image16"].data_ptr())
        if st:
            raise RuntimeError(lib.mbgb_last_error().decode())
        return s["image16"]
    o = s["out"]
    ctx.distance(s["scene"], s["points"].data_ptr(), s["detail"].data_ptr(), s["points"].shape[0],
                 o["distance"].data_ptr(), o["iterations"].data_ptr(), o["max_iter"].data_ptr(), s["prec"])
    return o


# What one pixel (or point) of each family takes: orbit iterations and operations of one
# iteration (the 21 of a Mandelbox iteration, the 27 of a power-8 Mandelbulb one, ...), counted
# on frames of these views; the layers' bytes per pixel.
_ORBIT = {"bulb": (80.0, 27.0), "box": (4000.0, 21.0), "deep": (5400.0, 27.0), "delta": (1300.0, 25.0),
          "menger": (1000.0, 20.0), "flight": (350.0, 27.0), "grad": (52.0, 135.0)}


def work(case) -> dict:
    kind = case["kind"]
    if kind == "batch":
        px = sum((W.FLIGHT_RESOLUTIONS[i % 4][0] // case["downscale"]) * (W.FLIGHT_RESOLUTIONS[i % 4][1] // case["downscale"])
                 for i in range(case["frames"]))
        its, ops = _ORBIT["flight"]
        return {"bytes": 23 * px, "flops": px * its * ops}
    if kind == "grad":
        px = case["frames"] * case["size"] ** 2
        its, ops = _ORBIT["grad"]
        return {"bytes": (24 + 72) * px, "flops": px * its * ops}
    if kind == "post":
        px = case["w"] * case["h"]
        # per direction and sample: the position, the plane projection, the slope
        return {"bytes": (12 + 4 + 2 + 3 + 6) * px, "flops": 15.0 * px * case["quality"] * (case["quality"] - 1)}
    if kind == "distance":
        return {"bytes": (32 + 13) * case["n"], "flops": case["n"] * 9.0 * (21.0 if case["scene"] == "box" else 27.0)}
    px = case["w"] * case["h"]
    its, ops = _ORBIT[case["scene"]]
    return {"bytes": (36 if kind == "host" else 23) * px, "flops": px * its * ops}


# --- the same values in plain 64-bit torch -------------------------------------------------

def _orbit64(scene, p, N, block=1 << 21):
    """Distance estimates of points [n, 3] (Mandelbox scale 2 or power-8 Mandelbulb), N
    iterations at most, in 64 bits; ended orbits leave the working set."""
    out = torch.zeros(p.shape[0], dtype=torch.float64, device=p.device)
    for b in range(0, p.shape[0], block):
        z = p[b:b + block].clone()
        c, at = z.clone(), torch.arange(b, b + z.shape[0], device=p.device)
        dr = torch.ones_like(z[:, 0])
        for _ in range(N):
            if scene == "box":
                z = z.clamp(-1.0, 1.0) * 2.0 - z
                r2 = (z * z).sum(1)
                k = torch.where(r2 < 0.25, 4.0, torch.where(r2 < 1.0, 1.0 / r2, 1.0))
                z = z * k[:, None] * 2.0 + c
                dr = dr * k * 2.0 + 1.0
            else:
                r = z.norm(dim=1)
                th, ph = 8.0 * torch.asin(z[:, 2] / r), 8.0 * torch.atan2(z[:, 1], z[:, 0])
                dr = 8.0 * r ** 7 * dr + 1.0
                z = torch.stack([th.cos() * ph.cos(), th.cos() * ph.sin(), th.sin()], 1) * (r ** 8)[:, None] + c
            r = z.norm(dim=1)
            end = r > (1024.0 if scene == "box" else 100.0)
            if bool(end.any()):
                e, f = r[end], dr[end]
                out[at[end]] = e / f if scene == "box" else 0.5 * e * e.log() / f
                z, c, dr, at = z[~end], c[~end], dr[~end], at[~end]
                if not z.shape[0]:
                    break
    return out


def _zbuffer64(case, seed):
    """The z-buffer: sphere tracing with the pixel footprint as threshold, the half-step
    bisection into its last hundredth, 1e20 where the ray leaves."""
    w, h, family = case["w"], case["h"], case["scene"]
    v = _view(3.5 if family == "bulb" else 20.0, seed)
    N, persp = (250 if family == "bulb" else 15), 2.0 * math.tan(math.radians(26.5)) / (w / h)
    a, b = math.radians(v["angle_alfa"]), math.radians(v["angle_beta"])
    rz = torch.tensor([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]], dtype=torch.float64)
    rx = torch.tensor([[1, 0, 0], [0, math.cos(b), -math.sin(b)], [0, math.sin(b), math.cos(b)]], dtype=torch.float64)
    x = ((torch.arange(w, dtype=torch.float64, device="cuda") / w - 0.5) * (w / h) * persp).repeat(h)
    y = ((torch.arange(h, dtype=torch.float64, device="cuda") / h - 0.5) * persp).repeat_interleave(w)
    d = torch.stack([x, torch.ones_like(x), y], 1) @ (rz @ rx).T.cuda()
    o = torch.tensor([v["view_point_x"], v["view_point_y"], v["view_point_z"]], dtype=torch.float64, device="cuda")
    foot = persp / w
    depth = torch.full((w * h,), 1e20, dtype=torch.float64, device="cuda")
    at, t = torch.arange(w * h, device="cuda"), torch.full((w * h,), 1e-15, dtype=torch.float64, device="cuda")
    step = t.clone()
    for _ in range(10000):   # march
        de, thr = _orbit64(family, o + d[at] * t[:, None], N), t * foot
        found = de.clamp(max=3.0) < thr
        if bool(found.any()):
            depth[at[found]] = _bisect64(family, o, d[at[found]], t[found], step[found] * 0.5, de[found], foot, N)
        step = de.clamp(max=3.0) - 0.5 * thr
        t = t + step
        keep = ~found & (t <= 50.0)
        at, t, step = at[keep], t[keep], step[keep]
        if not at.numel():
            break
    return depth.reshape(h, w)


def _bisect64(family, o, d, t, step, de, foot, N):
    t, done = t.clone(), torch.zeros_like(t, dtype=torch.bool)
    for _ in range(20):
        thr = t * foot
        done |= (de < thr) & (de > 0.99 * thr)
        t = torch.where(done, t, torch.where(de > thr, t + step, torch.where(de < 0.99 * thr, t - step, t)))
        de, step = _orbit64(family, o + d * t[:, None], N), step * 0.5
    return t


def exact(case, seed):
    """64-bit values where the path has such: distance estimates, and the z-buffer of the plain
    scenes. The shaded layers take palette entries by orbits of ten times the iterations, which
    round to other entries in any other arithmetic; the finite-difference estimate divides
    rounding errors by 1e-10; the deep zoom's rays differ by less than 64 bits hold."""
    if case["kind"] == "distance":
        points, _ = _points(case, seed)
        return {"distance": _orbit64(case["scene"], points, 15 if case["scene"] == "box" else 250),
                "iterations": None, "max_iter": None}
    if case["kind"] in ("still", "host") and case["scene"] in ("bulb", "box"):
        z = _zbuffer64(case, seed)
        out = dict.fromkeys([*_LAYERS] + ([] if case["kind"] == "still" else ["hit", "iters", "depth"]))
        out["zbuffer"] = z.float() if case["kind"] == "still" else z.cpu().numpy()
        if case["kind"] == "host":
            out["depth"] = out["zbuffer"]
        return out
    return None
