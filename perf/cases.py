"""Timing cases of the stereo library: what its users call, from one small pair to a large batch.

listed() names the cases, draw(rng) gives one more of the same ranges, prepare(case, seed) makes
a case's inputs on the GPU, run(state) is one pass through the public entry points, work(case) the
bytes and operations of a pass, and exact(case, seed) the pass's outputs in 64-bit arithmetic from
plain numpy and torch.

Inputs are generated on the GPU from the seed alone: rectified stereo pairs of a textured scene
(planes, slanted planes, or a sinusoidal surface with textureless patches), disparity and depth
maps with invalid pixels, and ORB keypoints of a rectified pair.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vx-rs_b200"))
import vx_sgm  # noqa: E402

DEVICE = "cuda"
PITCH = 512                    # row pitch of the images in bytes, as cudaMallocPitch rounds it
SERVED_SIZES = [(640, 480), (1242, 375), (1280, 720), (1920, 1080)]
BATCH_SIZES = [(320, 240), (640, 480), (1242, 375), (1280, 720)]
DISPARITIES = [64, 128, 192]
SERVED_BUDGET = 40 << 30


def listed():
    sgm = {"kind": "pair", "scene": "planes", "p1": 10, "p2": 120, "rx": 2, "ry": 2, "lr": True}
    return [
        # The smallest call: a preview-sized pair with the default window (9x7 census) and two paths.
        {**sgm, "name": "pair 320x240", "w": 320, "h": 240, "d": 64, "paths": 2, "rx": 4, "ry": 3, "lr": False},
        # A VGA camera pair, four paths and the left-right check: one synchronous call a frame.
        {**sgm, "name": "pair 640x480", "w": 640, "h": 480, "d": 64, "paths": 4},
        # A driving-benchmark frame (odd width, slanted ground), eight paths.
        {**sgm, "name": "pair 1242x375", "w": 1242, "h": 375, "d": 128, "paths": 8, "scene": "slanted"},
        # The largest request of the served workload as a call of its own.
        {**sgm, "name": "pair 1920x1080", "w": 1920, "h": 1080, "d": 192, "paths": 8},
        # Offline processing of many uneven pairs in one call (the benchmark's 64-pair mix).
        {"name": "batch of 64", "kind": "batch", "n": 64, "w": 0, "h": 0, "d": 0, "paths": 8, "mix": 3},
        # High-resolution frames in one call: the largest case.
        {"name": "batch of 2048x1536", "kind": "batch", "n": 8, "w": 2048, "h": 1536, "d": 256, "paths": 8, "mix": 0},
        # A burst of mixed requests at the server: host images in, host disparities out.
        {"name": "served burst", "kind": "served", "n": 16, "mix": 1},
        # The depth chain on one colour pair: gray conversion, disparity and depth, median, point cloud.
        {"name": "colour pair to cloud", "kind": "chain", "w": 640, "h": 480, "d": 64, "paths": 8},
        # The depth-map filters on a full-HD map.
        {"name": "median 1920x1080", "kind": "median", "w": 1920, "h": 1080, "radius": 2},
        {"name": "bilateral 1920x1080", "kind": "bilateral", "w": 1920, "h": 1080, "radius": 3, "ss": 5.0, "sd": 0.05},
        # Sparse stereo of a SLAM front end, and the frames of a recorded sequence in one call.
        {"name": "orb 2048", "kind": "orb", "nl": 2048, "nr": 2048},
        {"name": "orb 64 frames", "kind": "frames", "n": 64, "nl": 512, "nr": 512},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["pair", "batch", "served", "chain", "median", "bilateral", "orb", "frames"],
                       [8, 2, 1, 2, 3, 2, 2, 1])[0]
    if kind == "pair":
        window = rng.choice([(4, 3), (2, 2), (2, 2), (3, 2)])
        return {"kind": kind, "scene": rng.choice(["planes", "slanted", "surface"]), "w": log_int(rng, 160, 1920),
                "h": log_int(rng, 120, 1080), "d": rng.choice([16, 48, 64, 64, 100, 128, 128, 192, 256]),
                "paths": rng.choice([2, 4, 8, 8]), "p1": rng.choice([10, 10, 10, 15]),
                "p2": rng.choice([120, 120, 120, 120, 300]), "rx": window[0], "ry": window[1],
                "lr": rng.random() < 0.7}
    if kind == "batch":
        if rng.random() < 0.3:
            return {"kind": kind, "n": rng.randint(2, 8), "w": rng.randint(1024, 2048), "h": rng.randint(768, 1536),
                    "d": rng.choice([128, 192, 256]), "paths": rng.choice([4, 8]), "mix": 0}
        return {"kind": kind, "n": log_int(rng, 2, 64), "w": 0, "h": 0, "d": 0, "paths": rng.choice([4, 8, 8]),
                "mix": rng.randint(4, 1000)}
    if kind == "served":
        return {"kind": kind, "n": rng.randint(4, 20), "mix": rng.randint(2, 1000)}
    if kind == "chain":
        return {"kind": kind, "w": log_int(rng, 200, 1280), "h": log_int(rng, 150, 720),
                "d": rng.choice([64, 96, 128]), "paths": rng.choice([2, 4, 8])}
    if kind == "median":
        return {"kind": kind, "w": log_int(rng, 320, 2048), "h": log_int(rng, 240, 1536), "radius": rng.randint(1, 5)}
    if kind == "bilateral":
        return {"kind": kind, "w": log_int(rng, 320, 2048), "h": log_int(rng, 240, 1536), "radius": rng.randint(1, 6),
                "ss": rng.choice([2.0, 5.0]), "sd": rng.choice([0.05, 0.5, 2.0])}
    if kind == "orb":
        return {"kind": kind, "nl": log_int(rng, 256, 16384), "nr": log_int(rng, 256, 16384)}
    return {"kind": kind, "n": log_int(rng, 4, 64), "nl": log_int(rng, 128, 1024), "nr": log_int(rng, 128, 1024)}


# ---------------------------------------------------------------------------
# What a program creates once: the context and its handles.

@functools.lru_cache(maxsize=None)
def program():
    ctx = vx_sgm.Context(0)
    return {"ctx": ctx, "sgm": vx_sgm.SGMStereo(ctx), "filter": vx_sgm.DepthFilter(ctx),
            "color": vx_sgm.ColorConvert(ctx), "cloud": vx_sgm.DepthToCloud(ctx),
            "matcher": vx_sgm.StereoMatcher(ctx)}


@functools.lru_cache(maxsize=None)
def server():
    return vx_sgm.Server(program()["sgm"], program()["ctx"], memory_budget_bytes=SERVED_BUDGET, max_batch=32,
                         max_inflight_batches=2)


FORMATS = {torch.uint8: vx_sgm.FORMAT_U8, torch.float32: vx_sgm.FORMAT_F32, torch.int16: vx_sgm.FORMAT_I16}


def image(values, rgba=False):
    """A pitched device image holding `values` (H, W) or (H, W, 4): (texture, its pixels as a tensor)."""
    h, w = values.shape[:2]
    row = w * (4 if rgba else values.element_size())
    pitch = -(-row // PITCH) * PITCH
    buf = torch.zeros((h, pitch), dtype=torch.uint8, device=DEVICE)
    if rgba:
        view = buf[:, :row].view(h, w, 4)
        fmt = vx_sgm.FORMAT_RGBA8
    else:
        view = buf.view(values.dtype)[:, :w]
        fmt = FORMATS[values.dtype]
    view.copy_(values)
    texture = vx_sgm.Texture.wrap_device(program()["ctx"], buf.data_ptr(), pitch, w, h, fmt)
    texture.pixels = view          # the image lives as long as its texture
    return texture, view


def empty_image(h, w, dtype):
    return image(torch.zeros((h, w), dtype=dtype, device=DEVICE))


# ---------------------------------------------------------------------------
# Inputs

def generator(seed, salt=0):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEVICE)


def texture_image(g, h, w):
    """Uniform noise blurred with a Gaussian of 1.5 pixels, stretched to 0..255."""
    a = rand(g, h, w)
    r, sigma = 5, 1.5
    k = [math.exp(-(i * i) / (2 * sigma * sigma)) for i in range(-r, r + 1)]
    k = [v / sum(k) for v in k]
    for axis in (0, 1):
        n = a.shape[axis]
        i = torch.arange(n, device=DEVICE)
        out = torch.zeros_like(a)
        for j, v in enumerate(k):
            out += v * a.index_select(axis, (i + j - r).clamp(0, n - 1))
        a = out
    return (a - a.min()) * (255.0 / (a.max() - a.min()))


def disparity_map(g, scene, h, w, d):
    """Planes of constant (or, slanted, linear) disparity over a background, in [4, 0.9 d]."""
    lo, hi = min(4.0, 0.25 * d), 0.9 * d
    x = torch.arange(w, device=DEVICE, dtype=torch.float32)[None, :]
    y = torch.arange(h, device=DEVICE, dtype=torch.float32)[:, None]
    u = rand(g, 16, 8).cpu().tolist()
    out = torch.full((h, w), lo + (hi - lo) * 0.25 * u[0][0], device=DEVICE)
    if scene == "slanted":
        out = lo + (hi - lo) * (0.8 * y / h + 0.2 * x / w)
    for q in u[1:]:
        rw, rh = max(1.0, w * (0.1 + 0.4 * q[0])), max(1.0, h * (0.1 + 0.4 * q[1]))
        x0, y0 = q[2] * (w - rw), q[3] * (h - rh)
        inside = (x >= x0) & (x < x0 + rw) & (y >= y0) & (y < y0 + rh)
        level = lo + (hi - lo) * q[4]
        plane = torch.full((h, w), level, device=DEVICE)
        if scene == "slanted":
            plane = level + (x - x0) * (0.4 * q[5] - 0.2) + (y - y0) * (0.2 * q[6] - 0.1)
        out = torch.where(inside, plane, out)
    if scene == "surface":
        wave = lo + 0.5 * (hi - lo) + min(20.0, 0.25 * d) * torch.sin(x / 60.0) * torch.cos(y / 45.0)
        out = torch.where((y > 0.3 * h) & (y < 0.8 * h), wave, out)
    return out.round().clamp(0.0, d - 1.0)


def stereo_pair(seed, salt, scene, h, w, d):
    """(left, right) uint8 images with right(x, y) = left(x + disparity, y) plus noise of 2 levels."""
    g = generator(seed, salt)
    left = texture_image(g, h, w)
    disp = disparity_map(g, scene, h, w, d)
    if scene == "surface":         # a tenth of the image textureless
        u = rand(g, 2).cpu().tolist()
        ph, pw = max(1, int(h * 0.32)), max(1, int(w * 0.32))
        py, px = int(u[0] * (h - ph)), int(u[1] * (w - pw))
        left[py:py + ph, px:px + pw] = 128.0 + torch.randn(ph, pw, generator=g, device=DEVICE)
    x = torch.arange(w, device=DEVICE)[None, :] + disp.long()
    right = torch.gather(left, 1, x.clamp(max=w - 1))
    right = right + 2.0 * torch.randn(h, w, generator=g, device=DEVICE)
    right = torch.where(x < w, right, 255.0 * rand(g, h, w))
    return left.round().clamp(0, 255).to(torch.uint8), right.round().clamp(0, 255).to(torch.uint8)


def depth_values(seed, h, w):
    """A disparity map as the filters meet it: planes with noise, a quarter of the pixels invalid (-1)."""
    g = generator(seed, 77)
    d = disparity_map(g, "slanted", h, w, 128) + 0.3 * torch.randn(h, w, generator=g, device=DEVICE)
    return torch.where(rand(g, h, w) < 0.25, torch.full_like(d, -1.0), d.clamp(min=0.1))


def orb_keypoints(seed, salt, nl, nr, width=752, height=480):
    """Keypoints (x, y, response, level) and 256-bit descriptors of a rectified pair: four fifths of the
    left ones reappear on the right at x - disparity with row noise and flipped bits."""
    g = generator(seed, 1000 + salt)

    def positions(n):
        level = torch.where(rand(g, n) < 0.6, 0.0, (1 + 3 * rand(g, n)).floor().clamp(max=3))
        scale = 1.2 ** level
        x = (width * rand(g, n) / scale).floor() * scale
        y = (height * rand(g, n) / scale).floor() * scale
        return torch.stack([x, y, rand(g, n), level.to(torch.int32).view(torch.float32)], 1)

    def words(bits):
        w = (bits.view(-1, 8, 32).long() << torch.arange(32, device=DEVICE)).sum(2)
        return torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)

    left, right = positions(nl), positions(nr)
    lbits, rbits = rand(g, nl, 256) < 0.5, rand(g, nr, 256) < 0.5
    n = min(int(0.8 * nl), nr)
    src = torch.argsort(rand(g, nl))[:n]
    dst = torch.argsort(rand(g, nr))[:n]
    right[dst, 0] = left[src, 0] - (0.5 + 129.5 * rand(g, n))
    right[dst, 1] = left[src, 1] + 0.8 * torch.randn(n, generator=g, device=DEVICE)
    rbits[dst] = lbits[src] ^ (rand(g, n, 256) < 0.23 * rand(g, n, 1))
    return left.contiguous(), right.contiguous(), words(lbits), words(rbits)


def mixed(case, sizes):
    """The (w, h, d) of a mixed batch or burst: drawn from its own number, the same for every seed."""
    if not case["mix"]:
        return [(case["w"], case["h"], case["d"])] * case["n"]
    rng = np.random.default_rng(case["mix"])
    return [(*sizes[int(rng.integers(len(sizes)))], DISPARITIES[int(rng.integers(len(DISPARITIES)))])
            for _ in range(case["n"])]


def config(case):
    return vx_sgm.SGMStereoConfig(num_disparities=case["d"], p1=case.get("p1", 10), p2=case.get("p2", 120),
                                  census_radius_x=case.get("rx", 2), census_radius_y=case.get("ry", 2),
                                  num_paths=case["paths"], subpixel=True, lr_check=case.get("lr", True))


CHAIN_FOCAL, CHAIN_BASELINE = 500.0, 0.12
CHAIN_CLOUD = dict(min_depth=0.1, max_depth=10.0)


def colour_pair(case, seed):
    """RGBA images of the pair: the gray texture with a tint that varies over the image."""
    h, w = case["h"], case["w"]
    left, right = stereo_pair(seed, 0, "planes", h, w, case["d"])
    out = []
    for img in (left, right):
        f = img.float()
        out.append(torch.stack([(f * 0.9).round(), f, (f * 0.5 + 60.0).round().clamp(max=255),
                                torch.full_like(f, 255.0)], 2).to(torch.uint8))
    return out


# ---------------------------------------------------------------------------
# prepare and run

def prepare(case, seed):
    p = program()
    s = {"case": case, "p": p}
    kind = case["kind"]
    if kind == "pair":
        left, right = stereo_pair(seed, 0, case["scene"], case["h"], case["w"], case["d"])
        s["left"], s["right"] = image(left)[0], image(right)[0]
        s["out"], s["disparity"] = empty_image(case["h"], case["w"], torch.float32)
        s["out_i"], s["integer"] = empty_image(case["h"], case["w"], torch.int16)
        s["cfg"] = config(case)
    elif kind == "batch":
        shapes = mixed(case, BATCH_SIZES)
        scene = "planes" if case["mix"] else "surface"
        pairs = [stereo_pair(seed, i, scene, h, w, d) for i, (w, h, d) in enumerate(shapes)]
        s["left"], s["right"] = [image(a)[0] for a, _ in pairs], [image(b)[0] for _, b in pairs]
        s["out"] = [empty_image(h, w, torch.float32)[0] for w, h, _ in shapes]
        s["cfg"] = [config({**case, "d": d}) for _, _, d in shapes]
    elif kind == "served":
        shapes = mixed(case, SERVED_SIZES)
        pairs = [stereo_pair(seed, i, "planes", h, w, d) for i, (w, h, d) in enumerate(shapes)]
        s["pairs"] = [(a.cpu().numpy(), b.cpu().numpy()) for a, b in pairs]
        s["cfg"] = [config({"d": d, "paths": 8}) for _, _, d in shapes]
        s["server"] = server()
    elif kind == "chain":
        h, w = case["h"], case["w"]
        left, right = colour_pair(case, seed)
        s["rgba_l"], s["rgba_r"] = image(left, rgba=True)[0], image(right, rgba=True)[0]
        s["left"], s["gray_l"] = empty_image(h, w, torch.uint8)
        s["right"], s["gray_r"] = empty_image(h, w, torch.uint8)
        s["depth"], s["depth_px"] = empty_image(h, w, torch.float32)
        s["smooth"], s["smooth_px"] = empty_image(h, w, torch.float32)
        s["points"] = torch.zeros((h * w, 9), dtype=torch.float32, device=DEVICE)
        s["count"] = torch.zeros(1, dtype=torch.int32, device=DEVICE)
        s["cfg"] = config(case)
        s["camera"] = vx_sgm.CameraIntrinsics(CHAIN_FOCAL, CHAIN_FOCAL, w / 2, h / 2, w, h)
    elif kind in ("median", "bilateral"):
        s["in"] = image(depth_values(seed, case["h"], case["w"]))[0]
        s["out"], s["filtered"] = empty_image(case["h"], case["w"], torch.float32)
    else:
        frames = case.get("n", 1)
        sets = [orb_keypoints(seed, i, case["nl"], case["nr"]) for i in range(frames)]
        s["lk"], s["rk"], s["ld"], s["rd"] = (torch.cat([t[i] for t in sets]) for i in range(4))
        s["matches"] = torch.zeros((frames * case["nl"], 7), dtype=torch.int32, device=DEVICE)
        s["count"] = torch.zeros(frames, dtype=torch.int32, device=DEVICE)
        s["lo"] = np.arange(frames + 1, dtype=np.uint32) * case["nl"]
        s["ro"] = np.arange(frames + 1, dtype=np.uint32) * case["nr"]
        s["cfg"] = vx_sgm.StereoConfig()
    torch.cuda.synchronize()       # the library's stream does not wait for torch's
    return s


def match_outputs(s):
    m = s["matches"]
    return {"indices": m[:, :2], "disparity": m.view(torch.float32)[:, 2], "points": m.view(torch.float32)[:, 3:6],
            "count": s["count"]}


def run(s):
    case, p = s["case"], s["p"]
    ctx, kind = p["ctx"], case["kind"]
    if kind == "pair":
        p["sgm"].compute_disparity(ctx, s["left"], s["right"], s["out"], s["cfg"], output_i16=s["out_i"])
        return {"disparity": s["disparity"], "integer": s["integer"]}
    if kind == "batch":
        p["sgm"].compute_batch(ctx, s["left"], s["right"], s["out"], s["cfg"])
        return [t.pixels for t in s["out"]]
    if kind == "served":
        ids = [s["server"].submit(a, b, c, want_i16=False) for (a, b), c in zip(s["pairs"], s["cfg"])]
        return [s["server"].wait(i)[0] for i in ids]
    if kind == "chain":
        p["color"].rgba_to_gray(ctx, s["rgba_l"], s["left"])
        p["color"].rgba_to_gray(ctx, s["rgba_r"], s["right"])
        depth_map = p["sgm"].compute(ctx, s["left"], s["right"], s["cfg"], s["camera"], CHAIN_BASELINE,
                                     depth_out=s["depth"])
        p["filter"].apply_median(ctx, s["depth"], s["smooth"])
        k = s["camera"]
        p["cloud"].compute_device(ctx, s["smooth"], s["rgba_l"], k.fx, k.fy, k.cx, k.cy,
                                  vx_sgm.DepthToCloudConfig(**CHAIN_CLOUD), s["points"].data_ptr(),
                                  case["w"] * case["h"], s["count"].data_ptr())
        depth_map.texture.close()
        return {"gray_left": s["gray_l"], "gray_right": s["gray_r"], "depth": s["depth_px"],
                "smooth": s["smooth_px"], "points": s["points"][:, :3],
                "colour": s["points"].view(torch.int32)[:, 4], "count": s["count"]}
    if kind == "median":
        p["filter"].apply_median(ctx, s["in"], s["out"], vx_sgm.DepthMedianConfig(case["radius"]))
        return s["filtered"]
    if kind == "bilateral":
        p["filter"].apply_bilateral(ctx, s["in"], s["out"],
                                    vx_sgm.DepthFilterConfig(case["radius"], case["ss"], case["sd"]))
        return s["filtered"]
    if kind == "orb":
        p["matcher"].run_device(ctx, s["lk"].data_ptr(), case["nl"], s["rk"].data_ptr(), case["nr"],
                                s["ld"].data_ptr(), s["rd"].data_ptr(), s["cfg"], s["matches"].data_ptr(),
                                s["count"].data_ptr())
        return match_outputs(s)
    p["matcher"].run_frames_device(ctx, s["lo"], s["ro"], s["lk"].data_ptr(), s["rk"].data_ptr(), s["ld"].data_ptr(),
                                   s["rd"].data_ptr(), s["cfg"], s["matches"].data_ptr(), s["count"].data_ptr())
    return match_outputs(s)


def work(case):
    """Inputs read once and outputs written once; operations of the method at its least: census and cost
    one compare, XOR or popcount each, six for each path-pixel-disparity, one for each value a filter's
    window holds, four for each pair of keypoints' position tests."""
    kind = case["kind"]

    def sgm(w, h, d, paths, bits, out):
        return {"bytes": w * h * (2 + out), "flops": w * h * (2 * bits + 2 * d + 6 * d * paths + d)}

    def total(parts):
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}

    if kind == "pair":
        bits = (2 * case["rx"] + 1) * (2 * case["ry"] + 1) - 1
        return sgm(case["w"], case["h"], case["d"], case["paths"], bits, 6)
    if kind == "batch":
        return total([sgm(w, h, d, case["paths"], 24, 4) for w, h, d in mixed(case, BATCH_SIZES)])
    if kind == "served":
        return total([sgm(w, h, d, 8, 24, 4) for w, h, d in mixed(case, SERVED_SIZES)])
    if kind == "chain":
        px = case["w"] * case["h"]
        return total([sgm(case["w"], case["h"], case["d"], case["paths"], 24, 4),
                      {"bytes": px * (8 + 2 + 4 + 4 + 36), "flops": px * (2 * 5 + 9 + 6)}])
    if kind in ("median", "bilateral"):
        px, n = case["w"] * case["h"], (2 * case["radius"] + 1) ** 2
        return {"bytes": 8 * px, "flops": px * n * (1 if kind == "median" else 6)}
    frames = case.get("n", 1)
    return {"bytes": frames * (48 * (case["nl"] + case["nr"]) + 28 * case["nl"]),
            "flops": 4 * frames * case["nl"] * case["nr"]}


# ---------------------------------------------------------------------------
# The same outputs from plain numpy and torch

EXACT_PATH_PD = 6e8            # path-pixel-disparities that numpy runs within some 20 seconds


def census(img, rx, ry):
    """Descriptor bits (neighbour < centre, raster order, clamped coordinates) as uint64."""
    h, w = img.shape
    pad = np.pad(img, ((ry, ry), (rx, rx)), mode="edge")
    bits, b = np.zeros((h, w), np.uint64), 0
    for dy in range(2 * ry + 1):
        for dx in range(2 * rx + 1):
            if (dy, dx) != (ry, rx):
                bits |= (pad[dy:dy + h, dx:dx + w] < img).astype(np.uint64) << np.uint64(b)
                b += 1
    return bits


def sweep(cost, add, p1, p2, shifts):
    """One sweep of the path recurrence over the first axis of cost (T, D, N), for each shift of the last
    axis: every value is a 16-bit word, updated in place over d, as the method defines it."""
    t_n, d_n, n = cost.shape
    u16 = np.uint16
    k = len(shifts)
    prev = np.zeros((d_n, k, n), u16)
    m = np.zeros((k, n), u16)
    option = np.empty((d_n, k, n), u16)
    f = np.empty((k, n), u16)
    for t in range(t_n):
        if t:                      # each path's values come from its neighbour in the row before
            moved, m2 = np.zeros_like(prev), np.zeros_like(m)
            fresh = np.zeros((k, n), bool)
            for i, s in enumerate(shifts):
                a, b = max(s, 0), n + min(s, 0)
                moved[:, i, a:b] = prev[:, i, a - s:b - s]
                m2[i, a:b] = m[i, a - s:b - s]
                fresh[i, :a] = True
                fresh[i, b:] = True
            prev, m = moved, m2
        else:
            fresh = np.ones((k, n), bool)
        o3 = np.where(fresh, u16(0), m + u16(p2))
        np.add(prev[1:], u16(p1), out=option[:-1])
        option[-1] = 0xFFFF
        np.minimum(option, prev, out=option)
        np.minimum(option, o3, out=option)
        step = cost[t][:, None, :] + (u16(p1) - np.where(fresh, u16(0), m))
        f[:] = 0xFFFF
        for d in range(d_n):       # f = the value at d plus p1, which is the next d's option
            np.minimum(option[d], f, out=f)
            np.add(f, step[d], out=f)
            prev[d] = f
        prev -= u16(p1)
        m = prev.min(0)
        add(t, prev)


def exact_disparity(left, right, case):
    """(disparity as float64, integer disparity, both -1 where the left-right check fails)."""
    left, right = left.cpu().numpy(), right.cpu().numpy()
    h, w = left.shape
    d_n, paths = case["d"], case["paths"]
    rx, ry = case.get("rx", 2), case.get("ry", 2)
    p1, p2 = case.get("p1", 10), case.get("p2", 120)
    cl, cr = census(left, rx, ry), census(right, rx, ry)
    cost = np.full((h, d_n, w), 64, np.uint16)
    for d in range(min(d_n, w)):
        cost[:, d, d:] = np.bitwise_count(cl[:, d:] ^ cr[:, :w - d])
    total = np.zeros((h, d_n, w), np.uint16)
    across = np.ascontiguousarray(cost.transpose(2, 1, 0))
    down = [0] + ([1, -1] if paths == 8 else [])
    ways = [1, -1] if paths >= 4 else [1]
    for way in ways:
        def add_x(t, v):
            total[:, :, t if way > 0 else w - 1 - t] += v[:, 0].T

        def add_y(t, v):
            total[t if way > 0 else h - 1 - t] += v.sum(1, dtype=np.uint16)
        sweep(across[::way], add_x, p1, p2, [0])
        sweep(cost[::way], add_y, p1, p2, down)
    best = total.argmin(1)
    s = np.take_along_axis(total, best[:, None], 1)[:, 0].astype(np.float64)
    out = best.astype(np.float64)
    inner = (best > 0) & (best < d_n - 1)
    lo = np.take_along_axis(total, np.maximum(best - 1, 0)[:, None], 1)[:, 0].astype(np.float64)
    hi = np.take_along_axis(total, np.minimum(best + 1, d_n - 1)[:, None], 1)[:, 0].astype(np.float64)
    denom = 2.0 * (lo + hi - 2.0 * s)
    inner &= denom != 0
    out[inner] += (lo - hi)[inner] / denom[inner]
    if case.get("lr", True):
        rbest, rcost = np.zeros((h, w), np.int64), np.full((h, w), 1 << 30, np.int64)
        for d in range(min(d_n, w)):
            c = total[:, d, d:].astype(np.int64)
            better = c < rcost[:, :w - d]
            rbest[:, :w - d][better] = d
            rcost[:, :w - d][better] = c[better]
        xr = np.arange(w)[None, :] - best
        bad = (xr < 0) | (np.abs(best - np.take_along_axis(rbest, np.maximum(xr, 0), 1)) > 1)
        out[bad] = -1.0
        best = np.where(bad, -1, best)
    return out, best.astype(np.int16)


def windows(values, radius):
    """(n, H, W) values of the (2 radius + 1)^2 windows with clamped coordinates, raster order."""
    h, w = values.shape
    y, x = torch.arange(h, device=values.device), torch.arange(w, device=values.device)
    for dy in range(-radius, radius + 1):
        for dx in range(-radius, radius + 1):
            yield dy, dx, values[(y + dy).clamp(0, h - 1)][:, (x + dx).clamp(0, w - 1)]


def exact_median(values, radius):
    """The element count/2 of the window's sorted positive values, 0 where there is none."""
    stack = torch.stack([torch.where(v > 0, v, torch.full_like(v, math.inf)) for _, _, v in windows(values, radius)])
    count = (stack < math.inf).sum(0)
    out = stack.sort(0).values.gather(0, (count // 2)[None])[0]
    return torch.where(count > 0, out, torch.zeros_like(out))


def exact_bilateral(values, radius, ss, sd):
    c = values.double()
    total, weight = torch.zeros_like(c), torch.zeros_like(c)
    for dy, dx, v in windows(c, radius):
        wt = torch.where(v > 0, math.exp(-(dx * dx + dy * dy) / (2 * ss * ss)) *
                         torch.exp(-((v - c) ** 2) / (2 * sd * sd)), torch.zeros_like(c))
        total += v.clamp(min=0) * wt
        weight += wt
    out = torch.where(weight > 1e-8, total / weight, c)
    return torch.where(c > 0, out, torch.zeros_like(c))


def exact_matches(lk, rk, ld, rd, cfg):
    """Indices and triangulated points of the accepted matches, in left order, zeros after them."""
    def bits(words):
        return ((words[:, :, None].long() >> torch.arange(32, device=DEVICE)) & 1).flatten(1).float()

    lb, rb = bits(ld), bits(rd)
    best, dist = [], []
    for i in range(0, len(lk), 2048):
        a, k = lb[i:i + 2048], lk[i:i + 2048]
        ham = (a.sum(1)[:, None] + rb.sum(1)[None, :] - 2.0 * (a.double() @ rb.double().T)).long()
        disp = k[:, 0][:, None] - rk[:, 0][None, :]
        ok = ((k[:, 1][:, None] - rk[:, 1][None, :]).abs() <= cfg.max_epipolar) & \
            (disp >= cfg.min_disparity) & (disp <= cfg.max_disparity)
        key = torch.where(ok, ham * (1 << 24) + torch.arange(len(rk), device=DEVICE), 1 << 50).min(1).values
        best.append(key & ((1 << 24) - 1))
        dist.append(key >> 24)
    best, take = torch.cat(best), torch.cat(dist) <= cfg.max_hamming
    li = take.nonzero()[:, 0]
    ri = best[li]
    l, r = lk[li].double(), rk[ri].double()
    disp = l[:, 0] - r[:, 0]
    z = float(np.float32(cfg.fx)) * float(np.float32(cfg.baseline)) / disp
    n = len(lk)
    out = {"indices": torch.zeros((n, 2), dtype=torch.int32, device=DEVICE),
           "disparity": torch.zeros(n, dtype=torch.float64, device=DEVICE),
           "points": torch.zeros((n, 3), dtype=torch.float64, device=DEVICE),
           "count": torch.tensor([len(li)], dtype=torch.int32, device=DEVICE)}
    out["indices"][:len(li)] = torch.stack([li, ri], 1).int()
    out["disparity"][:len(li)] = disp
    out["points"][:len(li)] = torch.stack([z * (l[:, 0] - cfg.cx) / cfg.fx, z * (l[:, 1] - cfg.cy) / cfg.fy, z], 1)
    return out


def exact_chain(case, seed):
    gray = []
    for img in colour_pair(case, seed):
        c = img.float() / 255.0
        v = 0.299 * c[..., 0] + 0.587 * c[..., 1] + 0.114 * c[..., 2]
        gray.append((v.clamp(0, 1) * 255.0).round().to(torch.uint8))
    h, w = gray[0].shape
    disp = torch.from_numpy(exact_disparity(gray[0], gray[1], case)[0]).to(DEVICE)
    scale = float(np.float32(CHAIN_FOCAL) * np.float32(CHAIN_BASELINE))
    depth = torch.where(disp > 0, scale / disp.clamp(min=1e-9), torch.zeros_like(disp))
    smooth = exact_median(depth, 1)
    ok = (smooth >= float(np.float32(CHAIN_CLOUD["min_depth"]))) & (smooth <= CHAIN_CLOUD["max_depth"])
    y, x = ok.nonzero(as_tuple=True)
    z = smooth[y, x]
    points = torch.zeros((h * w, 3), dtype=torch.float64, device=DEVICE)
    points[:len(z)] = torch.stack([(x - w / 2) * z / CHAIN_FOCAL, (y - h / 2) * z / CHAIN_FOCAL, z], 1)
    return {"gray_left": None, "gray_right": None, "depth": depth, "smooth": smooth, "points": points,
            "colour": None, "count": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pair", "chain") and case["w"] * case["h"] * case["d"] * case["paths"] > EXACT_PATH_PD:
        return None
    if kind == "pair":
        left, right = stereo_pair(seed, 0, case["scene"], case["h"], case["w"], case["d"])
        disparity, integer = exact_disparity(left, right, case)
        return {"disparity": disparity, "integer": integer}
    if kind == "chain":
        return exact_chain(case, seed)
    if kind == "median":
        values = depth_values(seed, case["h"], case["w"])
        parts = []                 # by bands of rows, so that the sorted windows stay small
        r, h = case["radius"], case["h"]
        for y in range(0, h, 256):
            a, b = max(0, y - r), min(h, y + 256 + r)
            parts.append(exact_median(values[a:b], r)[y - a:min(h, y + 256) - a])
        return torch.cat(parts).double()
    if kind == "bilateral":
        return exact_bilateral(depth_values(seed, case["h"], case["w"]), case["radius"], case["ss"], case["sd"])
    if kind in ("orb", "frames"):
        sets = [orb_keypoints(seed, i, case["nl"], case["nr"]) for i in range(case.get("n", 1))]
        found = [exact_matches(*t, vx_sgm.StereoConfig()) for t in sets]
        return {k: torch.cat([f[k] for f in found]) for k in found[0]}
    return None
