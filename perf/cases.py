"""What this framework is timed on: whole frames, scene encoding and colour training, each through
the public Python entry points (gsr_b200.GpuScene, Renderer, ColorModel), over the range of sizes,
formats and options that the configurations, the tests and the benchmark of this repository use.

A case is a dict of plain values. `kind` says what is called:
  frame    Renderer.render, one view
  views    Renderer.render_views, several cameras in one frame
  host     Renderer.render_to_host, one view with its 8-bit image in pinned host memory
  learned  Renderer.render with a loaded colour model (the decode inside the preprocess)
  train    ColorModel(...), the training of a colour model, and its read-back
  encode   GpuScene(...), a host scene encoded into a GPU scene format

Scenes have the benchmark configurations' distributions (scenes.make_scene): means uniform in a
ball, log-scales N(-3.5, 0.7), opacity sigmoid(N(0, 1)), SH DC N(0, 0.5), higher bands N(0, 0.1).
They are drawn on the GPU, so that making a scene is quick.
"""
import math
import os
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "gaussian-splat-renderer_b200"))
import gsr_b200  # noqa: E402
from gsr_b200 import scenes  # noqa: E402


def _case(kind, n, width=0, height=0, **options):
    c = {"kind": kind, "n": n, "width": width, "height": height, "degree": 3, "fmt": "f32", "layout": "soa",
         "radius": 8.0, "views": 1, "uneven": False, "rgb8": False, "target": "rgba32f", "graph": False,
         "schedule": "auto", "list_mode": "binning", "tile": 16, "window": 0, "variable_sh": False}
    c.update(options)
    return c


def listed():
    return [
        # a viewer on a small scene with every setting at its default (no graph, the reference's
        # own test scene's degree 1): launches and host work count here
        _case("frame", 10_007, 641, 359, degree=1, radius=4.0) | {"name": "viewer_10k_360p"},
        # the 720p configuration: 100,000 gaussians, image and 8-bit image
        _case("frame", 100_000, 1280, 720, radius=5.0, rgb8=True, graph=True) | {"name": "frame_100k_720p"},
        # the 1080p orbit, one view a frame: the fp32 scene of 1.24 M gaussians
        _case("frame", 1_240_000, 1920, 1080, rgb8=True, graph=True) | {"name": "frame_1240k_1080p"},
        # the same orbit from the fp16 scene into the reference's default fp16 target, without graphs
        _case("frame", 1_240_000, 1920, 1080, fmt="f16", layout="split", target="rgba16f")
        | {"name": "frame_f16_1080p"},
        # the headline: eight 1080p views in one frame
        _case("views", 1_240_000, 1920, 1080, views=8, rgb8=True, graph=True, schedule="per-tile")
        | {"name": "views8_1240k_1080p"},
        # uneven cameras (256 x 256 to 1920 x 1080) in one frame, the queue rasterizer
        _case("views", 559_000, 0, 0, radius=6.0, views=24, uneven=True, rgb8=True, graph=True)
        | {"name": "views24_uneven_559k"},
        # 4K from 6 M gaussians: fp16 with a per-gaussian SH degree
        _case("frame", 6_000_000, 3840, 2160, radius=20.0, fmt="f16", layout="split", variable_sh=True, rgb8=True,
              graph=True) | {"name": "frame_6m_4k"},
        # the learned colour: latents decoded in the preprocess, a part of the gaussians on SH
        _case("learned", 1_240_000, 1920, 1080, graph=True) | {"name": "learned_1240k_1080p"},
        # the StopThePop window, 16 pending splats a pixel, on a ragged 8-bit (q8) scene
        _case("frame", 300_001, 1275, 717, radius=6.0, fmt="q8", layout="aos", window=16, graph=True)
        | {"name": "window16_300k_720p"},
        # a frame handed to the host: the call an exporter or a streaming server makes
        _case("host", 559_000, 1600, 900, radius=6.0, rgb8=True, graph=True) | {"name": "to_host_559k_900p"},
        # a colour model of a scene: the configuration's batch, a tenth of its 2,000 steps
        _case("train", 559_000, radius=6.0, steps=200, batch=65536) | {"name": "train_559k"},
        # a host scene into the q8 format with a per-gaussian SH degree
        _case("encode", 559_000, fmt="q8", layout="split", radius=6.0, variable_sh=True) | {"name": "encode_q8_559k"},
    ]


_SIZES = [(256, 256), (641, 359), (640, 480), (1023, 577), (1280, 720), (1600, 900), (1919, 1079), (1920, 1080)]


def draw(rng):
    """One more case of the listed ones' ranges: 10,000 to 2 M gaussians, 256 x 256 to 1080p, one
    to eight views, every format, list mode, tile shape and window size."""
    kind = rng.choices(["frame", "views", "host", "learned", "train", "encode"], [5, 3, 1, 1, 1, 1])[0]
    n = int(round(math.exp(rng.uniform(math.log(10_000), math.log(2_000_000)))))
    w, h = rng.choice(_SIZES)
    fmt, layout = rng.choice([("f32", "soa"), ("f32", "soa"), ("f32", "split"), ("f32", "aos"), ("f16", "split"),
                              ("f16", "aos"), ("q8", "split"), ("q8", "aos")])
    c = dict(radius=round(rng.uniform(4.0, 9.0), 2), fmt=fmt, layout=layout, degree=rng.choice([1, 2, 3, 3, 3]),
             graph=rng.random() < 0.6, rgb8=rng.random() < 0.5, variable_sh=rng.random() < 0.2)
    if kind == "train":
        return _case(kind, n, radius=c["radius"], steps=rng.randint(20, 200), batch=rng.choice([4096, 16384, 65536]),
                     degree=c["degree"])
    if kind == "encode":
        return _case(kind, n, **{k: c[k] for k in ("radius", "fmt", "layout", "degree", "variable_sh")})
    if kind == "learned":
        return _case(kind, n, w, h, **c)
    if kind == "host":
        return _case(kind, n, w, h, **{**c, "rgb8": True})
    c["list_mode"] = rng.choice(["binning", "binning", "binning", "global"])
    c["tile"] = rng.choice([16, 16, 16, 8, 32])
    if kind == "views":
        views = rng.randint(2, 8)
        return _case(kind, min(n, 1_240_000), w, h, **c, views=views, uneven=rng.random() < 0.5,
                     schedule=rng.choice(["auto", "per-tile"]))
    c["target"] = rng.choice(["rgba32f", "rgba32f", "rgba16f"])
    if rng.random() < 0.2:
        c["window"], n = rng.choice([1, 4, 8, 16]), min(n, 300_000)
    return _case(kind, n, w, h, **c)


# ---- inputs ----------------------------------------------------------------------------------------
def _gpu_arrays(case, seed):
    """The scene's activated float32 arrays on the GPU, in scenes.make_scene's distributions."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)
    n, K = case["n"], (case["degree"] + 1) ** 2

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    d = normal(n, 3)
    d /= d.norm(dim=1, keepdim=True).clamp_min(1e-20)
    r = case["radius"] * torch.rand(n, device="cuda", generator=g).pow(1.0 / 3.0)
    pos = torch.empty(n, 4, device="cuda")
    pos[:, :3] = d * r[:, None]
    pos[:, 3] = torch.sigmoid(normal(n))
    scales = torch.zeros(n, 4, device="cuda")
    scales[:, :3] = torch.exp(normal(n, 3) * 0.7 - 3.5)
    q = normal(n, 4)
    q /= q.norm(dim=1, keepdim=True).clamp_min(1e-20)
    sh = normal(n, K, 3) * 0.1
    sh[:, 0] *= 5.0
    if case["variable_sh"]:  # every degree in 0..degree as often, the bands above it zero
        deg = torch.randperm(n, device="cuda", generator=g) % (case["degree"] + 1)
        for k in range(1, K):
            sh[:, k] *= (deg >= math.isqrt(k)).float()[:, None]
    return pos, scales, q, sh


def _host_scene(case, seed):
    pos, scales, q, sh = _gpu_arrays(case, seed)
    return scenes.Scene(pos.cpu().numpy(), scales.cpu().numpy(), q.cpu().numpy(), sh.reshape(-1).cpu().numpy(),
                        case["degree"])


def _cameras(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    if case["uneven"]:  # the benchmark's resolutions, 40 to 90 degrees, from all around the scene
        sizes = [(c.width, c.height) for c in scenes.batched_cameras(case["views"], 2)]
        placed = scenes.batched_cameras(case["views"], int(rng.integers(1 << 30)))
        return [scenes.ViewerCamera(c.view, scenes.perspective_vk(rng.uniform(40.0, 90.0), w, h), c.model, w, h)
                for (w, h), c in zip(sizes, placed)]
    a0, out = rng.uniform(0.0, 2.0 * math.pi), []
    for k in range(case["views"]):
        a = a0 + 2.0 * math.pi * k / 300.0  # neighbours of a 300-frame orbit, 1.75 radii away
        far = 1.75 * case["radius"] if case["n"] < 4_000_000 else 1.5 * case["radius"]
        eye = (far * math.sin(a), 0.25 * case["radius"], far * math.cos(a))
        out.append(scenes.viewer_camera(eye, (0.0, 0.0, 0.0), case["width"], case["height"]))
    return out


def _gpu_scene(case, host):
    return gsr_b200.GpuScene(host, fmt=case["fmt"], layout=case["layout"],
                             sh_threshold=0.0 if case["variable_sh"] else -1.0)


class _Memory:
    """Device memory of the library as torch sees it (no copy); its owner lives as long as the tensor."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(pointer), False), "shape": tuple(shape), "typestr": typestr,
                                         "version": 2}


def _tensor(owner, pointer, shape, typestr):
    return torch.as_tensor(_Memory(owner, pointer, shape, typestr), device="cuda")


def _color_model(case, scene, seed):
    """A trained colour model as a program loads it: a checkpoint file with decoder weights of the
    trainer's initial scale, fp16 latents, and a tenth of the gaussians left to their SH colour."""
    rng = np.random.default_rng([int(seed), 5])
    params, at = np.zeros(gsr_b200.COLOR_MODEL_PARAMS, np.float32), 0
    for rows, cols, gain in ((48, 64, 6.0), (64, 8, 3.0), (11, 32, 6.0), (32, 32, 6.0), (32, 3, 3.0)):
        b = math.sqrt(gain / rows)
        params[at:at + rows * cols] = rng.uniform(-b, b, rows * cols)
        at += rows * cols + cols
    n = case["n"]
    latents = rng.standard_normal((n, 8), np.float32).astype(np.float16).view(np.uint16)
    fallback = rng.random(n) < 0.1
    latents[fallback, 7] = 0x7E00  # the marker: a half NaN in the last slot
    zeros = np.zeros_like(params)
    ck = {"count": n, "sh_degree": case["degree"], "step": 1, "options": {},
          "stats": {"gaussians": n, "fallback": int(fallback.sum()), "steps": 1, "sh_degree": case["degree"]},
          "params": params, "adam_m": zeros, "adam_v": zeros, "loss": np.zeros(1, np.float32), "latents": latents}
    fd, path = tempfile.mkstemp(suffix=".gsrc")
    os.close(fd)
    try:
        gsr_b200.write_color_checkpoint(path, ck)
        return gsr_b200.ColorModel.load(scene, path)
    finally:
        os.unlink(path)


def prepare(case, seed):
    host = _host_scene(case, seed)
    if case["kind"] == "encode":
        return {"case": case, "host": host}
    scene = _gpu_scene(case, host)
    if case["kind"] == "train":
        return {"case": case, "scene": scene, "seed": int(seed) % 65521 + 1}
    cameras = _cameras(case, seed)
    # the list starts large enough for the first frame and adapts from there
    renderer = gsr_b200.Renderer(scene, gsr_b200.Settings(
        budget_mb=2048, adaptive_initial_entries=8 * case["n"] * case["views"], rgb8=case["rgb8"],
        target=case["target"], use_graph=case["graph"], raster_schedule=case["schedule"], list_mode=case["list_mode"],
        tile_size=case["tile"], sort_window=case["window"]))
    state = {"case": case, "scene": scene, "renderer": renderer, "images": None}
    if case["kind"] == "learned":
        state["model"] = _color_model(case, scene, seed)
        renderer.set_color_model(state["model"])
    if case["kind"] == "views":
        state["cameras"] = gsr_b200.camera_array(cameras)
    else:
        state["camera"] = gsr_b200.to_c_camera(cameras[0])
    if case["kind"] == "host":
        state["out"] = torch.empty((case["height"], case["width"], 3), dtype=torch.uint8, pin_memory=True)
    return state


# ---- one pass --------------------------------------------------------------------------------------
def _images(state):
    """The renderer's image buffers (the same for every frame of one layout) as tensors."""
    if state["images"] is None:
        case, r = state["case"], state["renderer"]
        rgba, rgb, _, _ = r.image_pointers()
        pixels = sum(v.width * v.height for v in r.view_layouts())
        out = [_tensor(r, rgba, (pixels, 4), "<f4" if case["target"] == "rgba32f" else "<f2")]
        if case["rgb8"]:
            out.append(_tensor(r, rgb, (pixels, 3), "|u1"))
        state["images"] = tuple(out)
    return state["images"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "encode":
        scene = _gpu_scene(case, state["host"])
        d = scene.desc
        return [_tensor(scene, d.buffers[b], (int(d.buffer_bytes[b]) // 4,), "<i4") for b in range(4) if d.buffer_bytes[b]]
    if kind == "train":
        model = gsr_b200.ColorModel(state["scene"], steps=case["steps"], batch=case["batch"], seed=state["seed"])
        latents, params, loss = model.read()
        model.close()
        return {"latents": latents.view(np.float16), "params": params, "loss": loss}
    r = state["renderer"]
    if kind == "host":
        r.render_to_host(state["camera"], state["out"].numpy())
        return state["out"]
    if kind == "views":
        r.render_views(state["cameras"])
    else:
        r.render(state["camera"])
    return _images(state)


# ---- what a pass cannot do without -------------------------------------------------------------------
def _scene_bytes(case):
    """Bytes a gaussian of the scene format (a per-gaussian degree of 0..3 stores 7.5 of 16 coefficients)."""
    k = (case["degree"] + 1) ** 2
    if case["variable_sh"]:
        k = sum((d + 1) ** 2 for d in range(case["degree"] + 1)) / (case["degree"] + 1)
    return {"f32": 48 + 12 * k, "f16": 32 + 6 * k, "q8": 32 + 12 + 3 * (k - 1)}[case["fmt"]]


def work(case):
    n = case["n"]
    if case["kind"] == "encode":  # the host arrays across the link, the records written
        return {"bytes": n * (48 + 12 * (case["degree"] + 1) ** 2) + n * _scene_bytes(case), "flops": 0}
    if case["kind"] == "train":  # 12,000 multiply-adds a sample; the scene's SH read and the latents written
        return {"bytes": n * (12 * (case["degree"] + 1) ** 2 + 16), "flops": 24000.0 * case["batch"] * case["steps"]}
    pixels = case["width"] * case["height"] * case["views"]
    if case["uneven"]:  # the mean of the four resolutions
        pixels = case["views"] * (256 * 256 + 640 * 480 + 1280 * 720 + 1920 * 1080) // 4
    scene = _scene_bytes(case)
    if case["kind"] == "learned":  # the latent in the place of nine tenths of the colours
        geometry = 48 if case["fmt"] == "f32" else 32
        scene = geometry + 16 + 0.1 * (scene - geometry)
    image = (16 if case["target"] == "rgba32f" else 8) + (3 if case["rgb8"] else 0)
    # about 300 operations a gaussian and view, and 60 (pixel, splat) pairs a pixel of 16 operations
    return {"bytes": n * scene + pixels * image, "flops": 300.0 * n * case["views"] + 960.0 * pixels}


# ---- the same in 64 bits -------------------------------------------------------------------------------
def _stored(case, pos, scales, q, sh):
    """The values the scene format holds, in 64 bits."""
    if case["fmt"] == "f16":
        half = lambda x: x.half().double()  # noqa: E731
        q = half(q)
        q = q / q.norm(dim=1, keepdim=True)
        return torch.cat([pos[:, :3].double(), half(pos[:, 3:])], 1), half(scales), q, half(sh)
    return pos.double(), scales.double(), q.double(), sh.double()


def _sh_colour(degree, sh, d):
    x, y, z = d[:, 0:1], d[:, 1:2], d[:, 2:3]
    c = 0.28209479177387814 * sh[:, 0]
    if degree > 0:
        c = c - 0.4886025119029199 * (y * sh[:, 1] - z * sh[:, 2] + x * sh[:, 3])
    if degree > 1:
        xx, yy, zz, xy, yz, xz = x * x, y * y, z * z, x * y, y * z, x * z
        c = c + 1.0925484305920792 * (xy * sh[:, 4] - yz * sh[:, 5] - xz * sh[:, 7])
        c = c + 0.31539156525252005 * (2 * zz - xx - yy) * sh[:, 6] + 0.5462742152960396 * (xx - yy) * sh[:, 8]
        if degree > 2:
            c = c - 0.5900435899266435 * (y * (3 * xx - yy) * sh[:, 9] + x * (xx - 3 * yy) * sh[:, 15])
            c = c + 2.890611442640554 * xy * z * sh[:, 10] + 1.445305721320277 * z * (xx - yy) * sh[:, 14]
            c = c - 0.4570457994644658 * (4 * zz - xx - yy) * (y * sh[:, 11] + x * sh[:, 13])
            c = c + 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy) * sh[:, 12]
    return (c + 0.5).clamp_min(0.0)


def _project(case, seed):
    """The visible gaussians of the view, nearest first: pixel centre, conic, opacity, colour and
    the 16-pixel tile rectangle of three standard deviations."""
    pos, scales, q, sh = _stored(case, *_gpu_arrays(case, seed))
    cam = _cameras(case, seed)[0]
    w, h = case["width"], case["height"]
    view = torch.from_numpy(cam.view.astype(np.float64).reshape(4, 4)).cuda().T  # rows of the 4 x 4
    view = torch.diag(torch.tensor([1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device="cuda")) @ view
    R, eye = view[:3, :3], -(view[:3, :3].T @ view[:3, 3])
    tanx, tany = 1.0 / float(cam.proj[0]), 1.0 / abs(float(cam.proj[5]))
    t = pos[:, :3] @ R.T + view[:3, 3]
    keep = (t[:, 2] > 0.2) & (pos[:, 3] >= 1.0 / 255.0)
    pos, scales, q, sh, t = pos[keep], scales[keep, :3], q[keep], sh[keep], t[keep]
    r, x, y, z = q.unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                       2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                       2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    m = rot * scales[:, None, :]
    tz = t[:, 2]
    fx, fy = w / (2 * tanx), h / (2 * tany)
    tx = (t[:, 0] / tz).clamp(-1.3 * tanx, 1.3 * tanx) * tz
    ty = (t[:, 1] / tz).clamp(-1.3 * tany, 1.3 * tany) * tz
    J = torch.zeros(len(tz), 2, 3, dtype=torch.float64, device="cuda")
    J[:, 0, 0], J[:, 0, 2] = fx / tz, -fx * tx / (tz * tz)
    J[:, 1, 1], J[:, 1, 2] = fy / tz, -fy * ty / (tz * tz)
    a = J @ R @ m
    cov = a @ a.transpose(1, 2)
    c0, c1, c2 = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = c0 * c2 - c1 * c1
    mid = 0.5 * (c0 + c2)
    radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp_min(0.1))))
    cx = ((t[:, 0] / (tz * tanx) + 1) * w - 1) * 0.5
    cy = ((t[:, 1] / (tz * tany) + 1) * h - 1) * 0.5
    gx, gy = (w + 15) // 16, (h + 15) // 16
    rect = torch.stack([torch.trunc((cx - radius) / 16).clamp(0, gx), torch.trunc((cy - radius) / 16).clamp(0, gy),
                        torch.trunc((cx + radius + 15) / 16).clamp(0, gx),
                        torch.trunc((cy + radius + 15) / 16).clamp(0, gy)], 1)
    d = pos[:, :3] - eye
    colour = _sh_colour(case["degree"], sh, d / d.norm(dim=1, keepdim=True))
    data = torch.cat([cx[:, None], cy[:, None], (c2 / det)[:, None], (-c1 / det)[:, None], (c0 / det)[:, None],
                      pos[:, 3:4], colour], 1)
    order = torch.argsort(tz, stable=True)
    order = order[(det[order] != 0) & (rect[order, 2] > rect[order, 0]) & (rect[order, 3] > rect[order, 1])]
    return data[order], rect[order]


def exact(case, seed):
    """The image in 64 bits, tile by tile: front to back, alpha below 1/255 and power above 0 skipped,
    a pixel done when the next splat would bring its transmittance below 1e-4."""
    if case["kind"] != "frame" or case["window"] or case["fmt"] == "q8" or case["n"] > 1_500_000 \
            or case["width"] * case["height"] > 1920 * 1080:
        return None
    data, rect = _project(case, seed)
    w, h = case["width"], case["height"]
    image = torch.zeros((h + 15) // 16 * 16, (w + 15) // 16 * 16, 4, dtype=torch.float64, device="cuda")
    offset = torch.arange(16, dtype=torch.float64, device="cuda")
    for ty in range((h + 15) // 16):
        row = ((rect[:, 1] <= ty) & (rect[:, 3] > ty)).nonzero()[:, 0]
        row_data, row_rect = data[row], rect[row]
        py = (ty * 16 + offset)[:, None].expand(16, 16).reshape(1, -1)
        for tx in range((w + 15) // 16):
            tile = row_data[(row_rect[:, 0] <= tx) & (row_rect[:, 2] > tx)]
            px = (tx * 16 + offset)[None, :].expand(16, 16).reshape(1, -1)
            T = torch.ones(1, 256, dtype=torch.float64, device="cuda")
            rgb = torch.zeros(256, 3, dtype=torch.float64, device="cuda")
            alive = torch.ones(1, 256, dtype=torch.bool, device="cuda")
            for k in range(0, len(tile), 8192):
                s = tile[k:k + 8192]
                dx, dy = s[:, 0:1] - px, s[:, 1:2] - py
                power = -0.5 * (s[:, 2:3] * dx * dx + s[:, 4:5] * dy * dy) - s[:, 3:4] * dx * dy
                alpha = (s[:, 5:6] * torch.exp(power)).clamp_max(0.99)
                alpha = torch.where((power <= 0) & (alpha >= 1.0 / 255.0), alpha, 0.0)
                after = T * torch.cumprod(1 - alpha, 0)
                before = torch.cat([T, after[:-1]], 0)
                kept = (after >= 1e-4) & alive
                rgb += (alpha * before * kept).T @ s[:, 6:9]
                T = torch.where(kept, after, T).amin(0, keepdim=True)
                alive = alive & kept[-1:]
            image[ty * 16:ty * 16 + 16, tx * 16:tx * 16 + 16, :3] = rgb.reshape(16, 16, 3)
            image[ty * 16:ty * 16 + 16, tx * 16:tx * 16 + 16, 3] = (1 - T).reshape(16, 16)
    rgba = image[:h, :w].reshape(-1, 4).contiguous()
    return (rgba, None) if case["rgb8"] else (rgba,)
