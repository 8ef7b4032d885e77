"""The work that users of this package have it do, as cases that can be timed.

Each case goes through the public entry points (photon_tracer_b200 and the C
ABI under it) the way a program does: frames rendered on the device or into
host memory, scanlines, ray queries, a batch of scenes, and the two denoisers
with the network's training gradients. Sizes are those of the generators,
tests and benchmark of this repository, from one scanline to the 1024x1024,
64-sample room frame; draw() gives other sizes, sample counts and scenes of
the same ranges.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

import photon_tracer_b200 as pt
from photon_tracer_b200 import abi
from photon_tracer_b200.denoiser import WEIGHTS, trained
from photon_tracer_b200.unet import INPUT_CHANNELS, LAYERS, UNet, param_layout, primary_depth

# generator, look-from, look-at, vertical field of view, and for the work
# estimate: rays per sample, nodes / triangles / spheres / instances per ray
# (the traversal counters on each generator's own frame) and, roughly, the
# floating-point operations of a ray's shading and light sampling.
SCENES = {
    "spheres": (abi.PT_GEN_RANDOM_SPHERES, (13, 2, 3), (0, 0, 0), 20.0, (3.0, 5.0, 0.0, 2.5, 0.0), 250),
    "room": (abi.PT_GEN_ROOM_MESH, (0, 0, 3.3), (0, 0, 0), 40.0, (5.8, 4.7, 1.5, 0.5, 0.0), 250),
    "instances": (abi.PT_GEN_INSTANCES, (0, 35, 140), (0, 0, 0), 45.0, (2.6, 32.0, 5.1, 0.2, 6.4), 250),
    "textured": (abi.PT_GEN_TEXTURED, (0, 0, 0.3), (0, -0.15, -3.0), 62.0, (6.0, 4.0, 1.5, 0.5, 0.5), 300),
    "mesh_light": (abi.PT_GEN_MESH_LIGHT, (0, 0, 0.3), (0, -0.15, -3.0), 62.0, (6.0, 4.0, 1.5, 0.5, 0.0), 300),
}
BOX = ([-1.0, -1.0, -1.0], [1.0, 1.0, 1.0])  # ray origins inside the room


def listed():
    return [
        # a host program that still schedules scanlines itself and calls per row
        {"name": "row_spheres", "op": "row", "scene": "spheres", "param": 0, "width": 400, "height": 225, "spp": 16},
        # an interactive preview into host memory: the 400x225 sphere field at 16 samples
        {"name": "preview_spheres", "op": "host_frame", "scene": "spheres", "param": 0, "width": 400, "height": 225,
         "spp": 16},
        # the flagship: closed room with an 81,920-triangle mesh, a final frame left on the device
        {"name": "room_frame", "op": "frame", "scene": "room", "param": 6, "width": 1024, "height": 1024, "spp": 64,
         "extended": False},
        # what a denoiser is fed: a noisy 1080p frame with its guides and primary depth
        {"name": "room_guides", "op": "guides", "scene": "room", "param": 6, "width": 1920, "height": 1080, "spp": 4},
        # two-level traversal: 10,000 instances of three meshes
        {"name": "instances_frame", "op": "frame", "scene": "instances", "param": 10000, "width": 960, "height": 540,
         "spp": 16, "extended": False},
        # small scene, emissive triangles sampled as lights (the extended estimator)
        {"name": "mesh_light_extended", "op": "frame", "scene": "mesh_light", "param": 0, "width": 640, "height": 360,
         "spp": 16, "extended": True},
        # visibility / baking: many incoherent rays whose buffers stay on the device
        {"name": "closest_rays", "op": "closest", "scene": "room", "param": 6, "rays": 4194304},
        # a tool's line-of-sight checks: a few thousand host rays per call
        {"name": "any_rays_host", "op": "any_host", "scene": "room", "param": 4, "rays": 4099},
        # a service rendering many different small scenes at once
        {"name": "batch", "op": "batch", "scenes": 12, "side": 256, "spp": 4},
        # the edge-avoiding filter on a 1080p frame
        {"name": "atrous_1080p", "op": "atrous", "width": 1920, "height": 1080},
        # the learned denoiser on a 1080p frame
        {"name": "unet_1080p", "op": "unet", "width": 1920, "height": 1080},
        # one training batch of the learned denoiser: loss and every parameter's gradient
        {"name": "unet_grads", "op": "unet_grads", "batch": 16, "size": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["row", "host_frame", "frame", "frame", "frame", "guides", "closest", "any_host", "batch",
                     "atrous", "unet", "unet_grads"])
    if op in ("row", "host_frame", "frame", "guides"):
        kind = rng.choice(sorted(SCENES))
        width = _log(rng, 33, 1920)
        height = max(17, int(width / rng.uniform(1.0, 1.8)))
        if op == "row":
            spp = _log(rng, 1, 64)
        else:  # no more samples (two-level scenes: a sixteenth) than the largest listed frame
            most = (1 << 26 if op == "frame" else 1 << 23) // (16 if kind == "instances" else 2) // (width * height)
            spp = _log(rng, 1, max(1, min(64, most)))
        case = {"op": op, "scene": kind, "width": width, "height": height, "spp": spp,
                "param": {"room": rng.randint(2, 6), "spheres": rng.choice([0, _log(rng, 10, 2000)]),
                          "instances": _log(rng, 20, 10000)}.get(kind, 0)}
        if op == "frame":
            case["extended"] = rng.random() < 0.2
        return case
    if op == "closest":
        return {"op": op, "scene": rng.choice(["spheres", "room", "instances"]), "param": rng.randint(2, 6),
                "rays": _log(rng, 1000, 4 << 20)}
    if op == "any_host":
        return {"op": op, "scene": rng.choice(["spheres", "room", "instances"]), "param": rng.randint(2, 6),
                "rays": _log(rng, 1, 300000)}
    if op == "batch":
        return {"op": op, "scenes": rng.randint(2, 16), "side": rng.randint(100, 400), "spp": rng.choice([1, 2, 4])}
    if op in ("atrous", "unet"):
        width = _log(rng, 40, 1920)
        return {"op": op, "width": width, "height": max(9, int(width / rng.uniform(1.0, 1.8)))}
    return {"op": op, "batch": rng.randint(1, 16), "size": 8 * rng.randint(4, 16)}


# ---- inputs ------------------------------------------------------------------------------
def _scene(kind, param, seed):
    if kind == "instances" and param < 20:  # a ray query's small instanced scene
        param = 100 * param
    g = pt.Generated(SCENES[kind][0], seed=1 + seed % 1000, param=param)
    return g, pt.Scene(g)


def _camera(kind, width, height):
    _, look_from, look_at, vfov, _, _ = SCENES[kind]
    return pt.camera_look_at(look_from, look_at, vfov, width / height)


def _noisy_frame(seed, batch, height, width):
    """Colour, albedo, normal, depth, luminance variance and the clean colour
    of frames as a few-sample render gives them: flat-shaded regions, a sky
    without normals, multiplicative noise with a heavy tail."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(shape, device="cuda", generator=gen)

    cells = (batch, -(-height // 24), -(-width // 24))

    def spread(x, smooth=False):  # cells to pixels, channels last
        x = x if x.dim() == 4 else x[..., None]
        x = x.permute(0, 3, 1, 2)
        size = (cells[1] * 24, cells[2] * 24)
        x = F.interpolate(x, size=size, mode="bilinear", align_corners=False) if smooth else F.interpolate(x, size=size)
        return x[:, :, :height, :width].permute(0, 2, 3, 1).contiguous()

    albedo = spread(0.05 + 0.9 * rand(*cells, 3))
    normal = spread(F.normalize(rand(*cells, 3) - 0.5, dim=-1))
    sky = spread((rand(*cells) < 0.15).float()) > 0
    normal = torch.where(sky, torch.zeros_like(normal), normal)
    depth = torch.where(sky, torch.zeros_like(sky, dtype=torch.float32), spread(0.5 + 12 * rand(*cells)))
    light = spread(0.05 + 2 * rand(*cells, 3) ** 2, smooth=True)
    clean = light * albedo
    noise = torch.exp(0.7 * torch.randn((batch, height, width, 1), device="cuda", generator=gen) - 0.245)
    variance = (0.3 * clean.mean(-1) ** 2 * (0.25 + rand(batch, height, width))).contiguous()
    return ((clean * noise).contiguous(), albedo, normal, depth[..., 0].contiguous(), variance, clean.contiguous())


def _batch_items(case, seed):
    """Alternating rooms and sphere fields, every third one twice as wide, sample counts in three steps."""
    items = []
    for i in range(case["scenes"]):
        kind = "room" if i % 2 else "spheres"
        param = 2 + (i // 2) % 5 if kind == "room" else (50, 200, 800, 2000)[(i // 2) % 4]
        s = 1 + (seed * 31 + i) % 5000
        side = case["side"] * (2 if i % 3 == 2 else 1) + i
        g = pt.Generated(SCENES[kind][0], seed=s, param=param)
        items.append((g, _camera(kind, side, side), side, side, case["spp"] << (i % 3), s))
    return items


def _params(seed):
    """The network's parameters as training starts from: He-normal weights, zero biases."""
    rng = np.random.default_rng(seed)
    layout, total = param_layout()
    p = np.zeros(total, np.float32)
    for k, (w, shape, _, _) in enumerate(layout):
        n = int(np.prod(shape))
        fan_in = 9 * (INPUT_CHANNELS if k == 0 else shape[3])
        p[w:w + n] = rng.standard_normal(n, dtype=np.float32) * math.sqrt(2.0 / fan_in)
    return p


def _training(case, seed):
    size = case["size"]
    color, albedo, normal, depth, _, clean = _noisy_frame(seed, case["batch"], size, size)
    return torch.cat([color, albedo, normal, depth[..., None]], dim=-1).contiguous(), clean


def prepare(case, seed):
    op = case["op"]
    state = {"case": case, "op": op, "seed": seed}
    if op in ("row", "host_frame", "frame", "guides"):
        w, h = case["width"], case["height"]
        state["gen"], state["scene"] = _scene(case["scene"], case["param"], seed)
        state["camera"] = _camera(case["scene"], w, h)
        flags = abi.PT_FLAG_NEE_EXTENDED if case.get("extended") else 0
        state["settings"] = pt.Scene.settings(w, h, case["spp"], 10, seed=seed + 1, flags=flags)
        if op == "row":
            state["out"] = np.empty((w, 3), np.float32)
        if op in ("frame", "guides"):
            state["out"] = torch.empty((h, w, 3), dtype=torch.float32, device="cuda")
        if op == "guides":
            state["aux"] = torch.empty((h, w, 7), dtype=torch.float32, device="cuda")
    elif op in ("closest", "any_host"):
        state["gen"], state["scene"] = _scene(case["scene"], case["param"], seed)
        scale = {"room": 1.0, "spheres": 6.0, "instances": 60.0}[case["scene"]]
        box = [[scale * x for x in b] for b in BOX]
        state["rays"] = pt.generate_rays(seed + 1, box[0], box[1], case["rays"])
        if op == "closest":
            state["rays"] = torch.from_numpy(state["rays"]).cuda()
            state["hits"] = torch.empty((case["rays"], 6), dtype=torch.int32, device="cuda")
    elif op == "batch":
        state["batch"] = pt.Batch(_batch_items(case, seed), strategy=abi.PT_BATCH_ONE_LAUNCH)
    elif op == "atrous":
        w, h = case["width"], case["height"]
        color, albedo, normal, _, variance, _ = _noisy_frame(seed, 1, h, w)
        state["inputs"] = [color, albedo, normal, variance]
        state["out"] = torch.empty((h, w, 3), dtype=torch.float32, device="cuda")
        state["scratch"] = torch.empty(pt.load().pt_denoise_atrous_scratch_floats(w, h), dtype=torch.float32,
                                       device="cuda")
    elif op == "unet":
        w, h = case["width"], case["height"]
        color, albedo, normal, depth, _, _ = _noisy_frame(seed, 1, h, w)
        aux = torch.cat([albedo, normal, (color ** 2).mean(-1, keepdim=True)], dim=-1)
        state["frame"] = [color[0].contiguous(), aux[0].contiguous(), depth[0].contiguous()]
        state["net"] = trained()
    else:
        state["x"], state["target"] = _training(case, seed)
        state["net"] = UNet(seed=1)
        state["net"].set_params(_params(seed))
        state["grads"] = np.empty(state["net"].n_params, np.float32)
    return state


# ---- one pass ----------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return torch.cuda.current_stream().cuda_stream


def run(state):
    op, case = state["op"], state["case"]
    if op == "row":
        pt.render_row_linear(state["scene"], state["camera"], case["height"] // 2, case["width"], case["height"],
                             case["spp"], 10, state["out"], state["seed"] + 1)
        return state["out"]
    if op == "host_frame":
        image, _, rays = state["scene"].render(state["camera"], case["width"], case["height"], case["spp"], 10,
                                               seed=state["seed"] + 1)
        return [image, rays]
    if op == "frame":
        state["scene"].render_device(state["camera"], state["settings"], state["out"].data_ptr(), stream=_stream())
        return state["out"]
    if op == "guides":
        state["scene"].render_device(state["camera"], state["settings"], state["out"].data_ptr(),
                                     state["aux"].data_ptr(), stream=_stream())
        depth = primary_depth(state["scene"], state["camera"], case["width"], case["height"])
        return [state["out"], state["aux"], depth]
    if op == "closest":
        hits = state["hits"]
        state["scene"].trace_closest_device(state["rays"].data_ptr(), case["rays"], hits.data_ptr(), stream=_stream())
        return {"which": hits[:, 0:3], "where": hits.view(torch.float32)[:, 3:6]}
    if op == "any_host":
        return state["scene"].trace_any(state["rays"])
    if op == "batch":
        rays = state["batch"].render()
        return [rays] + [state["batch"].image(i) for i in range(case["scenes"])]
    if op == "atrous":
        color, albedo, normal, variance = state["inputs"]
        abi.check(pt.load().pt_denoise_atrous_device(
            case["width"], case["height"], _ptr(color), _ptr(albedo), _ptr(normal), _ptr(variance), _ptr(state["out"]),
            _ptr(state["scratch"]), ctypes.c_void_p(_stream())))
        return state["out"]
    if op == "unet":
        return state["net"].denoise(*state["frame"])
    loss = ctypes.c_float()
    grads = state["grads"]
    abi.check(pt.load().pt_unet_loss_grads(
        state["net"].h, case["batch"], case["size"], case["size"], _ptr(state["x"]), _ptr(state["target"]),
        ctypes.byref(loss), grads.ctypes.data_as(ctypes.c_void_p), None))
    return [float(loss.value), grads]


# ---- the work of a pass ------------------------------------------------------------------
def _scene_bytes(kind, param):
    """Roughly what the scene's trees and primitives hold, each read once."""
    if kind == "room":
        return 85 * 20 * 4 ** param
    return {"spheres": 100e3, "instances": 45e6, "textured": 1e6, "mesh_light": 20e3}[kind]


def _ray_flops(kind):
    _, nodes, tris, spheres, insts = SCENES[kind][4]
    # per node 4 boxes of 12 multiply/subtracts and 12 min/max; Moller-Trumbore, sphere and ray-transform operations
    return nodes * 96 + tris * 50 + spheres * 30 + insts * 36


def _frame_flops(kind, samples):
    return samples * SCENES[kind][4][0] * (_ray_flops(kind) + SCENES[kind][5])


def _unet_flops(batch, height, width):
    """Multiply-adds x 2 on the network's own channels (10 in, 3 out)."""
    total = 0.0
    for k, (cin, cout, level, _) in enumerate(LAYERS):
        cin = INPUT_CHANNELS if k == 0 else cin
        cout = 3 if k == len(LAYERS) - 1 else cout
        total += 18.0 * cin * cout * batch * (height >> level) * (width >> level)
    return total


def work(case):
    op = case["op"]
    if op in ("row", "host_frame", "frame", "guides"):
        px = case["width"] * (1 if op == "row" else case["height"])
        out = 44 if op == "guides" else 12
        return {"bytes": out * px + _scene_bytes(case["scene"], case["param"]),
                "flops": _frame_flops(case["scene"], px * case["spp"])}
    if op in ("closest", "any_host"):
        return {"bytes": (48 if op == "closest" else 25) * case["rays"] + _scene_bytes(case["scene"], case["param"]),
                "flops": case["rays"] * _ray_flops(case["scene"])}
    if op == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["scenes"]):
            kind = "room" if i % 2 else "spheres"
            px = (case["side"] * (2 if i % 3 == 2 else 1) + i) ** 2
            total["bytes"] += 12 * px + _scene_bytes(kind, 2 + (i // 2) % 5)
            total["flops"] += _frame_flops(kind, px * (case["spp"] << (i % 3)))
        return total
    if op == "atrous":
        px = case["width"] * case["height"]
        return {"bytes": 52 * px, "flops": 5 * 25 * 40 * px}  # 5 passes of 25 taps
    layout, n_params = param_layout()
    if op == "unet":
        px = case["width"] * case["height"]
        return {"bytes": 56 * px + 2 * n_params, "flops": _unet_flops(1, case["height"], case["width"])}
    px = case["batch"] * case["size"] ** 2
    return {"bytes": 52 * px + 6 * n_params, "flops": 3 * _unet_flops(case["batch"], case["size"], case["size"])}


# ---- the same outputs in 64 bits ---------------------------------------------------------
def _atrous_exact(color, albedo, normal, variance):
    """The filter of the reference's denoise.hpp: demodulate, five 5x5 passes with taps 1..16 apart, remodulate."""
    lum = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=color.device)
    color, albedo, normal, variance = (t[0].double() for t in (color, albedo, normal, variance))
    h, w = variance.shape
    base = albedo.clamp(min=0.01)
    light = color / base
    var = variance.clamp(min=0) / (albedo @ lum).clamp(min=0.01) ** 2
    length = normal.norm(dim=-1, keepdim=True)
    normal = torch.where(length > 1e-6, normal / length.clamp(min=1e-30), torch.zeros_like(normal))
    sky = (normal == 0).all(-1)

    def shifted(t, dy, dx):  # t at (y + dy, x + dx) for the pixels (ys, xs) where that lies inside
        ys, xs = slice(max(0, -dy), min(h, h - dy)), slice(max(0, -dx), min(w, w - dx))
        return t[max(0, dy):min(h, h + dy), max(0, dx):min(w, w + dx)], ys, xs

    for k in range(5):
        step = 1 << k
        blur, weight = torch.zeros_like(var), torch.zeros_like(var)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if abs(dy) < h and abs(dx) < w:
                    q, ys, xs = shifted(var, dy, dx)
                    c = (0.5 if dx else 1.0) * (0.5 if dy else 1.0)
                    blur[ys, xs] += c * q
                    weight[ys, xs] += c
        scale = 1 / (4 * torch.sqrt(blur / weight) + 1e-4)
        lp = light @ lum
        total, total_w, total_v = torch.zeros_like(light), torch.zeros_like(var), torch.zeros_like(var)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                if abs(dy * step) >= h or abs(dx * step) >= w:
                    continue
                lq, ys, xs = shifted(light, dy * step, dx * step)
                at = lambda t: shifted(t, dy * step, dx * step)[0]
                nd = (normal[ys, xs] * at(normal)).sum(-1).clamp(min=0) ** 64
                wgt = torch.where(sky[ys, xs], torch.ones_like(nd), nd) * (sky[ys, xs] == at(sky))
                da = ((albedo[ys, xs] - at(albedo)) ** 2).sum(-1)
                wgt = wgt * torch.exp(-da * 100 - (lp[ys, xs] - at(lp)).abs() * scale[ys, xs])
                wgt = wgt * (3 / 8, 1 / 4, 1 / 16)[abs(dx)] * (3 / 8, 1 / 4, 1 / 16)[abs(dy)]
                total[ys, xs] += wgt[..., None] * lq
                total_w[ys, xs] += wgt
                total_v[ys, xs] += wgt * wgt * at(var)
        light, var = total / total_w[..., None], total_v / total_w ** 2
    return light * base


def _unet_exact(params, x):
    """Log radiance [B, 3, H, W] of the network on [B, H, W, 10] guides; params as float64 tensors."""
    layout, _ = param_layout()

    def conv(i, t):
        off, shape, boff, cout = layout[i]
        wt = params[off:off + int(np.prod(shape))].view(shape).permute(0, 3, 1, 2)
        if i == 0:
            wt = wt[:, :INPUT_CHANNELS]
        y = 0
        tp = F.pad(t, (1, 1, 1, 1))
        h, w = t.shape[2], t.shape[3]
        for tap in range(9):  # nine matrix products, row by row of taps
            dy, dx = tap // 3, tap % 3
            y = y + torch.einsum("oc,bchw->bohw", wt[:, :, dy, dx], tp[:, :, dy:dy + h, dx:dx + w])
        y = y + params[boff:boff + cout].view(1, -1, 1, 1)
        return F.relu(y) if LAYERS[i][3] else y[:, :3]

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3)

    x = x.double()
    t = torch.cat([torch.log1p(x[..., :3].clamp(min=0)), x[..., 3:9], torch.log1p(x[..., 9:].clamp(min=0))], -1)
    t = t.permute(0, 3, 1, 2).contiguous()
    a1 = conv(1, conv(0, t))
    a3 = conv(3, conv(2, F.max_pool2d(a1, 2)))
    a5 = conv(5, conv(4, F.max_pool2d(a3, 2)))
    a7 = conv(7, conv(6, F.max_pool2d(a5, 2)))
    d2 = conv(9, conv(8, torch.cat([up(a7), a5], 1)))
    d1 = conv(11, conv(10, torch.cat([up(d2), a3], 1)))
    return conv(14, conv(13, conv(12, torch.cat([up(d1), a1], 1))))


def exact(case, seed):
    op = case["op"]
    if op == "atrous":
        color, albedo, normal, _, variance, _ = _noisy_frame(seed, 1, case["height"], case["width"])
        return _atrous_exact(color, albedo, normal, variance)
    if op == "unet":
        w, h = case["width"], case["height"]
        color, albedo, normal, depth, _, _ = _noisy_frame(seed, 1, h, w)
        x = torch.cat([color, albedo, normal, depth[..., None]], -1)
        x = F.pad(x.permute(0, 3, 1, 2), (0, -w % 8, 0, -h % 8), mode="replicate").permute(0, 2, 3, 1)
        with torch.no_grad():
            bits = np.load(WEIGHTS).astype(np.uint32) << 16  # the committed parameters are bfloat16 bits
            y = _unet_exact(torch.from_numpy(bits.view(np.float32)).cuda().double(), x)
        return torch.expm1(y).clamp(min=0)[0, :, :h, :w].permute(1, 2, 0).contiguous()
    if op == "unet_grads":
        x, target = _training(case, seed)
        p = torch.from_numpy(_params(seed)).cuda().double().requires_grad_(True)
        y = _unet_exact(p, x)
        loss = (y - torch.log1p(target.double().clamp(min=0)).permute(0, 3, 1, 2)).abs().mean()
        loss.backward()
        # whatever of the padding channels carries no gradient is zero here and there
        return [float(loss.item()), p.grad.cpu().numpy()]
    return None  # paths, hits and pixels follow from comparisons along each ray: no 64-bit form of the same values
