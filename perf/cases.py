"""The work a user of this framework has it do, as timed cases: the fused per-pixel render,
the print/scan of developed frames, each spatial stage (diffusion, scatter/halation, spatial
DIR, grain), the scanner post effects, the fitting chain forward and backward, and one whole
frame through the owner. Every case goes through the package's public calls
(film_juicer_b200.runtime / .fitting) on float32 planes and frames, the one data type the
boundary takes.

Sizes: frames from a 160x90 preview to 3840x2160, the common aspect ratios, odd and ragged
widths among them; the optics radii and sigmas follow the frame width as on a 35 mm gate.
Scenes are smooth fields plus fine texture over 12 stops, linear light.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import __graft_entry__

__graft_entry__.package()

from film_juicer_b200 import (abi, descriptors, fitting, frame_records, grain_plan, prepare as recipes,  # noqa: E402
                              runtime)

ROOT = os.path.dirname(os.path.abspath(__graft_entry__.__file__))
GATE_UM = 35000.0
RECIPES = ("print", "direct", "ektar100_endura", "vision3_500t_2383")
PRINT_RECIPES = ("print", "ektar100_endura", "vision3_500t_2383")
OPS = ("pixels", "scan", "post", "diffusion", "halation", "dir", "grain", "fit", "frame")


def listed():
    return [
        # the smallest call: the fused chain on a preview proxy, launch latency
        {"name": "preview_direct_160x90", "op": "pixels", "recipe": "direct", "width": 160, "height": 90,
         "components": 3},
        # a frame without spatial stages, RGBA, print route
        {"name": "pixels_print_1920x1080_rgba", "op": "pixels", "recipe": "print", "width": 1920, "height": 1080,
         "components": 4},
        # the print and scan of a developed 4K frame (the last stage of every print render)
        {"name": "scan_print_3840x2160", "op": "scan", "recipe": "print", "width": 3840, "height": 2160,
         "components": 3},
        # the same with the scanner's glare, lens blur and unsharp, at an odd size
        {"name": "post_print_1999x1333", "op": "post", "recipe": "vision3_500t_2383", "width": 1999, "height": 1333,
         "components": 3},
        # camera diffusion: a proxy frame of odd size (small radius) and the 4K frame
        {"name": "diffusion_1283x719", "op": "diffusion", "width": 1283, "height": 719, "radius": 6},
        {"name": "diffusion_3840x2160", "op": "diffusion", "width": 3840, "height": 2160, "radius": 19},
        # emulsion scatter and halation: a proxy frame of odd size and the 4K frame
        {"name": "halation_1283x719", "op": "halation", "width": 1283, "height": 719, "legacy": False},
        {"name": "halation_3840x2160", "op": "halation", "width": 3840, "height": 2160, "legacy": True},
        # the DIR couplers' spatial filter on the 4K frame
        {"name": "dir_3840x2160", "op": "dir", "width": 3840, "height": 2160, "tail_um": 200.0},
        # density-space grain of a 4K frame
        {"name": "grain_3840x2160", "op": "grain", "recipe": "print", "width": 3840, "height": 2160},
        # a fitting step on 16 crops: linear render and the gradient of 13 parameters
        {"name": "fit_16x512x512", "op": "fit", "recipe": "print", "width": 512, "height": 8192, "components": 3},
        # a whole 4K print frame through the owner: metering, diffusion, scatter/halation, spatial
        # DIR, print, scan. Grain is left to its own case: it draws whole particle counts, so a
        # last-bit difference ahead of it turns into another count.
        {"name": "frame_print_3840x2160", "op": "frame", "recipe": "print", "width": 3840, "height": 2160,
         "components": 3},
    ]


def draw(rng):
    op = rng.choice(OPS)
    aspect = rng.choice((16 / 9, 3 / 2, 4 / 3, 1.0, 2.39, 9 / 16))
    low = 160 * 90 if op == "pixels" else 640 * 360
    pixels = math.exp(rng.uniform(math.log(low), math.log(3840 * 2160 if op != "fit" else 16 * 512 * 512)))
    width = max(64, int(math.sqrt(pixels * aspect)))
    height = max(64, min(int(pixels / width), 4096 * 2160 // width))
    if rng.random() < 0.5:
        width -= width % 8  # half of the frames have the round widths cameras and hosts use
    case = {"op": op, "width": width, "height": height}
    if op in ("pixels", "scan", "post", "fit", "frame", "grain"):
        case["recipe"] = rng.choice(RECIPES if op in ("pixels", "scan", "post", "fit") else PRINT_RECIPES)
    if op in ("pixels", "scan", "post", "fit", "frame"):
        case["components"] = rng.choice((3, 3, 4))
    if op == "diffusion":
        case["radius"] = max(1, int(round(width * rng.choice((0.003, 0.005, 0.008)))))
    if op == "halation":
        case["legacy"] = rng.random() < 0.5
    if op == "dir":
        case["tail_um"] = rng.choice((100.0, 200.0, 300.0))
    return case


# ---------------------------------------------------------------------------
# What a program keeps: recipes laid out once on the device, the grain noise, one owner
# ---------------------------------------------------------------------------
_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _recipe(name):
    path = os.path.join(ROOT, "tests", "golden", "recipe_%s.npz" % name)
    return _keep(("recipe", name), lambda: recipes.PreparedRecipe.load(path))


def _device_recipe(name):
    return _keep(("device", name), lambda: runtime.DeviceRecipe(recipes.HostRecord(_recipe(name))))


def _noise():
    return _keep("noise", grain_plan.synthetic_noise)


def _device_noise():
    return _keep("device noise", lambda: runtime.DeviceNoise(_noise().record))


def _owner():
    return _keep("owner", runtime.Owner)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _fields(case, seed, count):
    """`count` smooth fields in [0, 1] with fine texture, (count, H, W) float32 on the GPU."""
    h, w = case["height"], case["width"]
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, :] / w
    y = torch.arange(h, device="cuda", dtype=torch.float32)[:, None] / w
    out = torch.empty((count, h, w), device="cuda", dtype=torch.float32)
    for k in range(count):
        a = rng.uniform(0, 2 * math.pi)
        f = math.cos(a) * (x - 0.5) + math.sin(a) * (y - 0.5 * h / w)
        for _ in range(8):
            cx, cy, s = rng.uniform(0, 1), rng.uniform(0, h / w), rng.uniform(0.02, 0.15)
            gx, gy = torch.exp(-((x - cx) / s) ** 2 / 2), torch.exp(-((y - cy) / s) ** 2 / 2)
            f = torch.addcmul(f, gy * float(rng.uniform(-1, 1)), gx)
        lo, hi = f.min(), f.max()
        f = 0.02 + 0.96 * (f - lo) / (hi - lo) + 0.01 * torch.randn((h, w), device="cuda", generator=gen)
        out[k] = f.clamp_(0.0, 1.0)
    return out


def _scene(case, seed):
    """(H, W, components) linear Rec.709: luminance 2^-8 .. 2^4, moderate chroma."""
    f = _fields(case, seed, 3)
    lum = torch.exp2(-8.0 + 12.0 * f[0])
    hue, chroma = 2 * math.pi * f[1], 0.3 * f[2]
    rgb = torch.empty((case["height"], case["width"], case.get("components", 3)), device="cuda", dtype=torch.float32)
    for c, phase in enumerate((0.0, 2.1, 4.2)):
        rgb[..., c] = lum * (1.0 + chroma * torch.cos(hue + phase))
    if rgb.shape[2] == 4:
        rgb[..., 3] = f[1]
    return rgb


def _exposure(case, seed):
    """Camera exposure planes R, G, B, linear, over 12 stops."""
    return torch.exp2(-8.0 + 12.0 * _fields(case, seed, 3))


def _density(case, seed):
    """Developed film densities C, M, Y above base."""
    return 0.05 + 2.1 * _fields(case, seed, 3)


def _components(pixel_um):
    """Nine exponential components of a warm bloom filter: core 8 um, halo 40 um, bloom 150 um."""
    c = abi.FjDiffusionComponents()
    groups = ((8.0, 1.5, (0.5, 0.5), 0.55), (40.0, 2.0, (0.36, 0.33, 0.31), 0.30),
              (150.0, 2.5, (0.34, 0.27, 0.21, 0.18), 0.15))
    tint = {1: ((0.9, 1.0, 1.1), (0.98, 1.0, 1.02), (1.12, 1.0, 0.88))}
    i = 0
    for g, (center, spread, weights, share) in enumerate(groups):
        n = len(weights)
        for k, wt in enumerate(weights):
            t = 2.0 * k / (n - 1) - 1.0
            c.lambda_px[i] = center * spread ** t / pixel_um
            for ch, field in enumerate((c.red_weights, c.green_weights, c.blue_weights)):
                field[i] = share * wt * (tint[g][ch][k] if g in tint else 1.0)
            i += 1
    return c


def prepare(case, seed):
    op, w, h = case["op"], case["width"], case["height"]
    px = GATE_UM / w
    s = {"case": case}
    if op == "pixels":
        s["recipe"], s["src"] = _device_recipe(case["recipe"]), _scene(case, seed)
        s["dst"] = torch.empty_like(s["src"])
    elif op in ("scan", "post"):
        s["recipe"], s["density"] = _device_recipe(case["recipe"]), _density(case, seed)
        s["dst"] = torch.empty((h, w, case["components"]), device="cuda")
        s["src"] = _scene(case, seed + 1) if case["components"] == 4 else None
        if op == "post":
            s["post"] = descriptors.scanner_post_record(
                glare_percent=0.3, glare_blur_sigma_px=max(0.5, 4.0 * w / 3840), lens_blur_sigma_px=0.8,
                unsharp_sigma_px=0.7, unsharp_amount=0.7)
            need = runtime.load_library().fjb_scanner_post_scratch_bytes(w, h)
            s["scratch"] = torch.empty(int(need) // 4, device="cuda")
    elif op == "diffusion":
        s["components"], s["fraction"] = _components(px), 0.12
        s["src"] = _exposure(case, seed)
        s["dst"] = torch.empty_like(s["src"])
    elif op == "halation":
        s["record"] = recipes.scatter_halation_record(px, legacy=case["legacy"])
        s["src"] = _exposure(case, seed)
        s["work"] = torch.empty_like(s["src"])
        need = runtime.load_library().fjb_scatter_halation_scratch_bytes(w, h)
        s["scratch"] = torch.empty(int(need) // 4, device="cuda")
    elif op == "dir":
        record = descriptors.spatial_dir_record(px, w, h, tail_um=case["tail_um"])
        s["filter"] = runtime.DirFilter(record, w, h)
        s["src"] = 0.9 * _fields(case, seed, 3)
        s["dst"] = torch.empty_like(s["src"])
    elif op == "grain":
        s["recipe"], s["noise"] = _device_recipe(case["recipe"]), _device_noise()
        a = _recipe(case["recipe"]).arrays
        layers = [[a["density_layers"][:, i, c] for c in range(3)] for i in range(3)]
        inp = grain_plan.GrainInput(render_extent=(0, 0, w, h), full_frame_extent=(0, 0, w, h), pixel_size_um=px,
                                    frame_time=float(seed % 1000), layer_curves=layers)
        s["record"] = grain_plan.visual_grain_record(inp, grain_plan.plan(inp), grain_plan.GrainCoefficients(),
                                                     curves_cmy=a["density_rgb"])
        s["src"] = _density(case, seed)
        s["work"] = torch.empty_like(s["src"])
        need = runtime.load_library().fjb_visual_grain_scratch_bytes(w, h)
        s["scratch"] = torch.empty((int(need) + 3) // 4, device="cuda")
    elif op == "fit":
        s["recipe"], s["src"] = _device_recipe(case["recipe"]), _scene(case, seed)
        theta = fitting.default_theta(s["recipe"]).to(torch.float32)
        theta[[0, 1, 2, 12]] += torch.tensor([0.1, -0.05, 0.08, -0.1])
        s["theta"] = theta.requires_grad_(True)
        s["cotangent"] = (2.0 / (3 * h * w)) * (_fields(case, seed + 2, 3) - 0.2)
    elif op == "frame":
        s["record"] = frame_records.FrameRecord(_recipe(case["recipe"]), w, h, grain=False, auto_exposure=True,
                                                recipe_hash=1 + RECIPES.index(case["recipe"]))
        s["owner"], s["src"] = _owner(), _scene(case, seed)
        s["dst"] = torch.empty_like(s["src"])
    else:
        raise ValueError(op)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "pixels":
        s["recipe"].render(s["src"], s["dst"])
        return s["dst"]
    if op == "scan":
        s["recipe"].render_from_density(tuple(s["density"]), s["src"], s["dst"])
        return s["dst"]
    if op == "post":
        runtime.render_from_density_post(s["recipe"], s["post"], 0x51A2E, (0, 0), tuple(s["density"]), s["dst"],
                                         src=s["src"], scratch=s["scratch"])
        return s["dst"]
    if op == "diffusion":
        runtime.diffusion(s["components"], case["radius"], s["fraction"], tuple(s["src"]), tuple(s["dst"]))
        return s["dst"]
    if op == "halation":
        s["work"].copy_(s["src"])  # the stage works in place on the frame's carrier
        runtime.scatter_halation(s["record"], tuple(s["work"]), scratch=s["scratch"])
        return s["work"]
    if op == "dir":
        s["filter"].apply(tuple(s["src"]), tuple(s["dst"]))
        return s["dst"]
    if op == "grain":
        s["work"].copy_(s["src"])  # the stage works in place on the frame's densities
        runtime.visual_grain(s["recipe"], s["record"], tuple(s["work"]), s["noise"], scratch=s["scratch"])
        return s["work"]
    if op == "fit":
        s["theta"].grad = None
        rgb = fitting.chain(s["theta"], s["recipe"], s["src"])
        rgb.backward(s["cotangent"])
        return {"rgb": rgb.detach(), "gradient": s["theta"].grad}
    s["owner"].render(s["record"], s["src"], s["dst"])
    return s["dst"]


# Arithmetic per pixel of the path's parts, in floating-point operations: the spectral
# integral (81 wavelengths: three-term density, exponential, three sums), the camera's 16-tap
# table, the scanner's tricubic cell, curves and colour.
_PRINT, _CAMERA, _SCAN = 81 * 13, 150, 450


def _recursive_flops(gaussians):
    return gaussians * 2 * 2 * 7  # forward and backward, rows and columns, a third-order step


def work(case):
    op, n = case["op"], case["width"] * case["height"]
    comps = case.get("components", 3)
    printing = _PRINT if case.get("recipe") in PRINT_RECIPES else 0
    if op == "pixels":
        return {"bytes": 8 * comps * n, "flops": (_CAMERA + printing + _SCAN) * n}
    if op == "scan":
        return {"bytes": (12 + 4 * comps + (4 if comps == 4 else 0)) * n, "flops": (printing + _SCAN) * n}
    if op == "post":
        return {"bytes": (12 + 4 * comps + (4 if comps == 4 else 0)) * n, "flops": (printing + _SCAN + 3 * 100) * n}
    if op == "diffusion":
        # a real transform there and back of each channel
        return {"bytes": 24 * n, "flops": 3 * 5 * math.log2(n) * n}
    if op == "halation":
        # three tails and the core on three channels, three bounces on two of them
        return {"bytes": 24 * n, "flops": _recursive_flops(3 * 4 + 2 * 3) * n}
    if op == "dir":
        return {"bytes": 24 * n, "flops": _recursive_flops(3 * 4) * n}
    if op == "grain":
        return {"bytes": 24 * n, "flops": 9 * 60 * n}
    if op == "fit":
        return {"bytes": (8 * comps + 24) * n, "flops": 3 * (_CAMERA + printing + _SCAN) * n}
    return {"bytes": 8 * comps * n,
            "flops": (_CAMERA + _PRINT + _SCAN + 15 * math.log2(n) + _recursive_flops(18 + 12)) * n}


# ---------------------------------------------------------------------------
# The spatial stages in 64 bits. The chains through the scanner's table (pixels, scan, post,
# fit, frame) have no value outside this package: the table is built by the library. Grain is
# a draw.
# ---------------------------------------------------------------------------
def _mirror(n, pad, whole, device="cuda"):
    """Indices of a line of n samples extended by `pad` on both sides by reflection about the
    end samples (whole) or about the edges between samples."""
    i = torch.arange(-pad, n + pad, device=device)
    if n == 1:
        return torch.zeros_like(i)
    period = 2 * (n - 1) if whole else 2 * n
    i = i.remainder(period)
    return torch.where(i < n, i, (period if whole else period - 1) - i)


def _exact_diffusion(case, seed):
    r, w, h = case["radius"], case["width"], case["height"]
    comp, f = _components(GATE_UM / w), 0.12
    src = _exposure(case, seed).double()
    d = torch.arange(-r, r + 1, device="cuda", dtype=torch.float64)
    rho = torch.sqrt(d[:, None] ** 2 + d[None, :] ** 2)
    iy, ix = _mirror(h, r, True), _mirror(w, r, True)
    out = torch.empty_like(src)
    for c, weights in enumerate((comp.red_weights, comp.green_weights, comp.blue_weights)):
        psf = sum(weights[k] * torch.exp(-rho / comp.lambda_px[k]) / (2 * math.pi * comp.lambda_px[k] ** 2)
                  for k in range(9))
        psf = psf / psf.sum()
        ext = src[c][iy][:, ix]
        size = tuple(ext.shape)
        big = torch.zeros(size, device="cuda", dtype=torch.float64)
        big[:2 * r + 1, :2 * r + 1] = psf
        conv = torch.fft.irfft2(torch.fft.rfft2(ext) * torch.fft.rfft2(big), s=size)[2 * r:, 2 * r:]
        out[c] = (1 - f) * src[c] + f * conv
    return out


def _fir(x, taps, dim):
    r = (len(taps) - 1) // 2
    ext = x.index_select(dim, _mirror(x.shape[dim], r, False))
    return sum(float(t) * ext.narrow(dim, k, x.shape[dim]) for k, t in enumerate(taps))


def _recursion(x, b, a, start, factored=None):
    """y_n = b x_n + a1 y_{n-1} + a2 y_{n-2} + a3 y_{n-3} along the first axis, the history
    before it being `start`; factored (h, g, t): the same filter as a first- and a
    second-order section."""
    y = torch.empty_like(x)
    if factored is not None:
        h, g, t = factored
        s1, s2, s3 = start.clone(), start.clone(), torch.zeros_like(start)
        for n in range(x.shape[0]):
            s1 = s1 + h * (x[n] - s1)
            s3 = t * s3 + g * (s1 - s2)
            s2 = s2 + s3
            y[n] = s2
        return y
    y1 = y2 = y3 = start
    for n in range(x.shape[0]):
        v = torch.addcmul(b * x[n], a[2], y3)
        v = torch.addcmul(v, a[1], y2)
        v = torch.addcmul(v, a[0], y1)
        y[n] = v
        y1, y2, y3 = v, y1, y2
    return y


def _exact_halation(case, seed):
    rec = recipes.scatter_halation_record(GATE_UM / case["width"], legacy=case["legacy"])
    planes = list(_exposure(case, seed).double())

    def blur(plane, g, columns):
        if g.kind == abi.FJ_HALATION_IDENTITY:
            return plane
        if g.kind == abi.FJ_HALATION_FIR_REFLECT:
            return _fir(plane, list(g.fir_weights)[:2 * g.radius + 1], 0 if columns else 1)
        one = lambda v: torch.tensor(float(v), device="cuda", dtype=torch.float64)  # noqa: E731
        x = plane.flip(0) if columns else plane.t()
        x = x.contiguous()
        k = [float(v) for v in g.yvv]
        fac = tuple(k[:3]) if g.kind == abi.FJ_HALATION_YVV_REPLICATE_FACTORED else None
        a = [one(v) for v in k[1:4]]
        y = _recursion(x, k[0], a, x[0], fac)
        z = _recursion(y.flip(0).contiguous(), k[0], a, y[-1], fac)
        return z if columns else z.flip(0).t()

    def gauss(plane, g):
        return blur(blur(plane, g, False), g, True)

    amps = [float(np.float32(v)) for v in (0.1633, 0.6496, 0.1870)]
    for c in range(3):
        ch, x, a = rec.channels[c], planes[c], float(rec.scatter_amount)
        tw = float(ch.tail_weight)
        tail = sum(amp * gauss(x, ch.tail[i]) for i, amp in enumerate(amps)) if tw > 0 else 0.0
        x = (1 - a) * x + a * ((1 - tw) * gauss(x, ch.core) + tw * tail)
        s = float(ch.total_strength)
        if s != 0.0:
            x = x + s * sum(float(rec.bounce_weights[b]) * gauss(x, ch.bounce[b]) for b in range(rec.bounce_count))
            if rec.renormalize:
                x = x / (1 + s)
        planes[c] = x
    return torch.stack(planes)


def _exact_dir(case, seed):
    w, h = case["width"], case["height"]
    rec = descriptors.spatial_dir_record(GATE_UM / w, w, h, tail_um=case["tail_um"])
    src = (0.9 * _fields(case, seed, 3)).double()

    def blur(x, g, dim):
        if g.reference_operator == abi.FJ_DIR_OPERATOR_IDENTITY:
            return x
        sigma = float(g.sigma_px)
        if g.reference_operator == abi.FJ_DIR_OPERATOR_FIR_REFLECT:
            t = np.arange(-g.radius, g.radius + 1, dtype=np.float64)
            taps = np.exp(-t * t / (2 * sigma * sigma))
            return _fir(x, taps / taps.sum(), dim)
        pad = int(14 * sigma) + 64
        ext = x.index_select(dim, _mirror(x.shape[dim], pad, False)).movedim(dim, 0).contiguous()
        a = [torch.tensor(float(v), device="cuda", dtype=torch.float64) for v in g.feedback]
        for _ in range(2):
            ext = _recursion(ext, float(g.feedforward), a, ext[0]).flip(0).contiguous()
        return ext.narrow(0, pad, x.shape[dim]).movedim(0, dim)

    return sum(float(rec.components[k].weight) * blur(blur(src, rec.components[k], 2), rec.components[k], 1)
               for k in range(rec.component_count))


def exact(case, seed):
    with torch.no_grad():
        if case["op"] == "diffusion":
            return _exact_diffusion(case, seed)
        if case["op"] == "halation":
            return _exact_halation(case, seed)
        if case["op"] == "dir":
            return _exact_dir(case, seed)
    return None
