"""The work that users of the library have it do, as measured cases: frames
and batches through RawConverter, the pyramid denoise on its own, calibration
gradients, burst registration and fusion, and noise-model measurement.

A case is a dict of plain values. prepare() makes its inputs on the GPU from a
seed and the objects that a user's program keeps (converter, detector, output
buffers); run() is one pass through the public entry points; exact() gives the
same outputs from float64 PyTorch. Sizes are those of the repository's
workloads, tests and benchmark, and generic ones between them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch
import torch.nn.functional as F

import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import adjoint, registration, scene

DEV = "cuda"
F64 = torch.float64

# Workload noise: gain (electrons per DN) and read noise (DN) of the sensor,
# by the ISO the frame was taken at.
GAIN = {200: (0.8, 3.0), 400: (0.8, 3.0), 800: (1.5, 4.0), 1600: (2.0, 5.0)}


def listed():
    return [
        # a thumbnail-sized crop, one call: launches and serial kernels count
        {"name": "frame_256x192_f16", "kind": "frame", "w": 256, "h": 192, "levels": 3, "storage": "f16",
         "iso": 400, "post": False},
        # the FP32 plain path, as a tool that wants the reference's arithmetic calls it
        {"name": "frame_1024x768_f32", "kind": "frame", "w": 1024, "h": 768, "levels": 4, "storage": "f32",
         "iso": 200, "post": False},
        # one 12 MP capture to display sRGB: the camera application's call
        {"name": "frame_4032x3024_f16_srgb", "kind": "frame", "w": 4032, "h": 3024, "levels": 5, "storage": "f16",
         "iso": 1600, "post": True},
        # a directory of 12 MP captures, six frames a call: throughput
        {"name": "batch_6x4032x3024_f16", "kind": "batch", "sizes": "4032x3024,4032x3024,4032x3024,4032x3024,"
         "4032x3024,4032x3024", "levels": 5, "iso": 1600},
        # captures of four sensors in one call (ragged sizes, 12 and 14 bits): the largest
        {"name": "batch_mixed_4_sensors_f16", "kind": "batch", "sizes": "4032x3024,6000x4000,5472x3648,8368x5584",
         "levels": 5, "iso": 800},
        # the denoiser alone on a YCbCr image of odd size, FP32 planes
        {"name": "denoise_1367x1025_f32", "kind": "denoise", "w": 1367, "h": 1025, "levels": 5, "storage": "f32",
         "iso": 800},
        # the denoiser alone, FP16 planes, a half-resolution 12 MP image
        {"name": "denoise_2016x1512_f16", "kind": "denoise", "w": 2016, "h": 1512, "levels": 5, "storage": "f16",
         "iso": 1600},
        # one frame of a calibration run: loss and the gradient of 32 parameters
        {"name": "calibrate_2048x1536", "kind": "calibrate", "w": 2048, "h": 1536, "levels": 5, "iso": 800},
        # features of one Bayer channel of a 12 MP frame
        {"name": "detect_2016x1512", "kind": "detect", "w": 2016, "h": 1512, "features": 1500},
        # the registration of an 8-frame burst, two channels, features detected
        {"name": "register_8_frames", "kind": "register", "w": 2016, "h": 1512, "features": 1500, "n": 8},
        # pyramid fusion of that burst's 12 MP frames
        {"name": "fuse_8x4032x3024", "kind": "fuse", "w": 4032, "h": 3024, "n": 8, "levels": 5, "robustness": 100.0,
         "storage": "f16"},
        # the noise models of a 12 MP frame: the raw model and the level-0 YCbCr model
        {"name": "noise_model_4032x3024", "kind": "noise", "w": 4032, "h": 3024, "storage": "f16", "iso": 800},
    ]


def draw(rng):
    def size(lo, hi, even):
        """Width and height, log-uniform in the pixel count."""
        px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        aspect = rng.choice([4 / 3, 3 / 2, 16 / 9, 1.0])
        w, h = int(math.sqrt(px * aspect)), int(math.sqrt(px / aspect))
        return (w & ~1, h & ~1) if even else (w, h)

    def levels(w, h):  # at least 24 patches on the coarsest level
        n = 5
        while n > 1 and ((w >> (n - 1)) // 8) * ((h >> (n - 1)) // 8) < 24:
            n -= 1
        return n

    kind = rng.choice(["frame", "frame", "frame", "batch", "denoise", "denoise", "calibrate", "detect", "register",
                       "fuse", "noise"])
    iso = rng.choice(sorted(GAIN))
    if kind == "frame":
        w, h = size(20e3, 12.2e6, True)
        n = levels(w, h)
        storage = rng.choice(["f16", "f16", "f32"])
        post = n == 5 and storage == "f16" and rng.random() < 0.4
        return {"kind": kind, "w": w, "h": h, "levels": n, "storage": storage, "iso": iso, "post": post}
    if kind == "batch":
        sizes = []
        while len(sizes) < 8:
            w, h = size(300e3, 24e6, True)
            if sum(a * b for a, b in sizes) + w * h > 90e6:
                break
            sizes.append((w, h))
            if len(sizes) >= 2 and rng.random() < 0.2:
                break
        n = min(levels(w, h) for w, h in sizes)
        return {"kind": kind, "sizes": ",".join("%dx%d" % s for s in sizes), "levels": n, "iso": iso}
    if kind == "denoise":
        w, h = size(20e3, 12.2e6, False)
        return {"kind": kind, "w": w, "h": h, "levels": levels(w, h), "storage": rng.choice(["f16", "f32"]),
                "iso": iso}
    if kind == "calibrate":
        w, h = size(20e3, 3.1e6, True)
        return {"kind": kind, "w": w, "h": h, "levels": levels(w, h), "iso": iso}
    if kind in ("detect", "register"):
        w, h = size(300e3, 3.2e6, False)
        c = {"kind": kind, "w": w, "h": h, "features": min(rng.choice([500, 1000, 1500, 2000]), w * h // 1000)}
        return c if kind == "detect" else dict(c, n=rng.randint(2, 8))
    if kind == "fuse":
        w, h = size(200e3, 12.2e6, False)
        return {"kind": kind, "w": w, "h": h, "n": rng.randint(2, 8), "levels": rng.randint(3, 5),
                "robustness": rng.choice([0.0, 25.0, 100.0]), "storage": rng.choice(["f16", "f32"])}
    w, h = size(200e3, 12.2e6, True)
    return {"kind": kind, "w": w, "h": h, "storage": rng.choice(["f16", "f32"]), "iso": iso}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _scene(w, h, gen, blobs=0.0):
    """A linear RGB scene in [0, 1], (3, h, w): three octaves of smooth noise
    and 20 rectangles, mean 18%; with blobs, that many small squares and
    crosses per megapixel for a feature detector."""
    img = torch.full((3, h, w), 0.5, device=DEV)
    for o in range(3):
        per = max(w, h) / 6.0 / 2 ** o
        gw, gh = int(w / per) + 4, int(h / per) + 4
        lat = torch.rand((1, 3, gh, gw), device=DEV, generator=gen) * 2 - 1
        img += 0.45 * 0.5 ** o * F.interpolate(lat, size=(h, w), mode="bicubic", align_corners=False)[0]
    img.clamp_(0, 1)
    r = torch.rand((20, 8), generator=torch.Generator().manual_seed(int(torch.randint(1 << 30, (1,), device=DEV,
                                                                                       generator=gen)))).tolist()
    for a in r:
        rw, rh = int(w * (0.05 + 0.2 * a[0])) + 1, int(h * (0.05 + 0.2 * a[1])) + 1
        x, y = int(a[2] * max(1, w - rw)), int(a[3] * max(1, h - rh))
        top = 0.9 if a[4] < 0.15 else 0.02
        for c in range(3):
            img[c, y:y + rh, x:x + rw] = top + a[5 + c] * ((1.0 if top > 0.5 else 0.9) - top)
    if blobs:
        for r in (1, 2, 3, 5, 7, 10):
            imp = (torch.rand((1, 1, h, w), device=DEV, generator=gen) < blobs / 6e6).float()
            val = imp * (0.2 + 2.8 * torch.rand((1, 1, h, w), device=DEV, generator=gen))
            m = F.max_pool2d(val, 2 * r + 1, 1, r)[0]
            img = torch.where(m > 0, m * img.mean(), img)
    return (img * (0.18 / img.mean())).clamp_(0, 1)


def _mosaic(rgb):
    """RGGB samples of a (3, h, w) image."""
    out = rgb[1].clone()
    out[0::2, 0::2] = rgb[0, 0::2, 0::2]
    out[1::2, 1::2] = rgb[2, 1::2, 1::2]
    return out


def _noisy(m, wl, gen):
    """Poisson-Gaussian sensor noise: the raw DN, int16 storage of uint16."""
    e = torch.poisson(m.clamp(min=0) * ((wl.white - wl.black) * wl.gain), generator=gen)
    dn = e / wl.gain + wl.read * torch.randn(m.shape, device=DEV, generator=gen) + wl.black
    return dn.round().clamp(0, wl.white).to(torch.int32).to(torch.int16)


def _workload(w, h, levels, iso, bits=12):
    gain, read = GAIN[iso]
    white, black = (4095, 512) if bits == 12 else (16383, 2048)
    return scene.Workload("case", w, h, levels=levels, black=black, white=white, gain=gain, read=read, iso=iso)


def _params(wl, post=False):
    p = scene.make_params(wl)
    if post:  # the reference application's display settings
        p.rgb_conversion.contrast, p.rgb_conversion.saturation = 1.05, 1.0
        p.rgb_conversion.tone_curve_slope, p.rgb_conversion.local_tone_mapping = 3.5, 1
        p.ltm.eps, p.ltm.shadows, p.ltm.highlights = 0.01, 1.0, 1.0
        for k, d in enumerate((1.0, 1.2, 2.0)):
            p.ltm.detail[k] = d
    return p


def _frames(case, seed):
    """[(workload, raw, clean scene)] of a frame, batch or calibration case."""
    if case["kind"] == "batch":
        sizes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    else:
        sizes = [(case["w"], case["h"])]
    out = []
    for i, (w, h) in enumerate(sizes):
        gen = _gen(seed * 64 + i)
        wl = _workload(w, h, case["levels"], case["iso"], 12 if i % 2 == 0 else 14)
        rgb = _scene(w, h, gen)
        out.append((wl, _noisy(_mosaic(rgb), wl, gen), rgb))
    return out


def _ycc_input(case, seed):
    """A noisy YCbCr image (h, w, 4) and its gradient (h, w, 2): sensor noise
    of the case's ISO as the level-0 model gives it, blurred |gradients|."""
    w, h = case["w"], case["h"]
    gen = _gen(seed * 64 + 1)
    wl = _workload(w, h, case.get("levels", 5), case["iso"])
    p = _params(wl)
    rgb = 0.1 + 0.9 * _scene(w, h, gen)
    m = torch.tensor(_matrices(p)[0], device=DEV, dtype=torch.float32)
    ycc = torch.einsum("ij,jhw->ihw", m, rgb)
    nlf = p.pyramid_nlf[0]
    for c in range(3):
        sd = (nlf.a[c] + nlf.b[c] * ycc[0].clamp(min=0)).sqrt()
        ycc[c] = ycc[c] + sd * torch.randn((h, w), device=DEV, generator=gen)
    y = F.avg_pool2d(F.pad(ycc[:1][None], (2, 2, 2, 2), mode="replicate"), 5, 1)[0, 0]
    grad = torch.stack([torch.diff(y, dim=1, append=y[:, -1:]).abs() * 2,
                        torch.diff(y, dim=0, append=y[-1:]).abs() * 2], -1)
    ycc = torch.cat([ycc, torch.zeros((1, h, w), device=DEV)]).permute(1, 2, 0)
    dt = torch.float16 if case["storage"] == "f16" else torch.float32
    return wl, p, ycc.to(dt).contiguous(), grad.to(dt).contiguous()


def _warp(img, H):
    """img (c, h, w) seen through H (reference -> frame pixels), bilinear."""
    h, w = img.shape[-2:]
    Hi = torch.tensor(np.linalg.inv(H), device=DEV, dtype=torch.float32)
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                          torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    d = Hi[2, 0] * x + Hi[2, 1] * y + Hi[2, 2]
    u = (Hi[0, 0] * x + Hi[0, 1] * y + Hi[0, 2]) / d
    v = (Hi[1, 0] * x + Hi[1, 1] * y + Hi[1, 2]) / d
    grid = torch.stack([2 * u / max(w - 1, 1) - 1, 2 * v / max(h - 1, 1) - 1], -1)[None]
    return F.grid_sample(img[None], grid, mode="bilinear", padding_mode="border", align_corners=True)[0]


def _burst_raws(case, seed, n):
    """n raw frames of one textured scene, twice the case's channel size."""
    w, h = 2 * case["w"], 2 * case["h"]
    gen = _gen(seed * 64 + 2)
    wl = _workload(w, h, 5, 800)
    ref = _scene(w, h, gen, blobs=1500.0)
    Hs = scene.burst_homographies(n, w, h, seed)
    return wl, [_noisy(_mosaic(ref if i == 0 else _warp(ref, Hs[i])), wl, gen) for i in range(n)]


def _view(t, channels):
    return g.ImageView(C.c_void_p(t.data_ptr()), t.shape[1], t.shape[0], channels,
                       g.F16 if t.dtype == torch.float16 else g.F32, t.stride(0) * t.element_size())


def _half(case):
    return case.get("storage", "f16") == "f16"


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("frame", "batch"):
        fr = _frames(case, seed)
        dt = torch.float16 if _half(case) else torch.float32
        s["conv"] = g.RawConverter(0)
        s["raws"] = [r for _, r, _ in fr]
        s["params"] = [_params(wl, case.get("post", False)) for wl, _, _ in fr]
        s["outs"] = [torch.empty((wl.height, wl.width, 4), dtype=dt, device=DEV) for wl, _, _ in fr]
    elif kind == "denoise":
        _, p, ycc, grad = _ycc_input(case, seed)
        out = torch.empty_like(ycc)
        s.update(conv=g.RawConverter(0), p=p, ycc=ycc, grad=grad, out=out,
                 views=(_view(ycc, 4), _view(grad, 2), _view(out, 4)))
    elif kind == "calibrate":
        (wl, raw, rgb), = _frames(case, seed)
        s.update(conv=g.RawConverter(0), raw=raw, p=_params(wl),
                 target=(0.1 + 0.9 * rgb).permute(1, 2, 0).contiguous())
    elif kind in ("detect", "register"):
        n = case.get("n", 1)
        wl, raws = _burst_raws(case, seed, n)
        surf = registration.SURF(case["w"], case["h"], max_features=case["features"], nOctaves=4, nOctaveLayers=2,
                                 hessianThreshold=0.02)
        s["surf"] = surf
        for f, raw in enumerate(raws):
            planes = surf.raw_channels(raw, wl.pattern, float(wl.black), float(wl.white), 4.0)
            torch.cuda.synchronize()
            if kind == "detect":
                s["plane"] = planes[1]
            else:
                surf.detect_slot(planes[1], 2 * f, sync=True)
                surf.detect_slot(planes[3], 2 * f + 1, sync=True)
    elif kind == "fuse":
        w, h, n = case["w"], case["h"], case["n"]
        gen = _gen(seed * 64 + 3)
        ref = _scene(w, h, gen)
        s["Hs"] = [H.astype(np.float32) for H in scene.burst_homographies(n, w, h, seed)]
        dt = torch.float16 if _half(case) else torch.float32
        s["frames"] = []
        for i in range(n):
            f = ref if i == 0 else _warp(ref, np.asarray(s["Hs"][i], np.float64))
            f = f + 0.01 * torch.randn(f.shape, device=DEV, generator=gen)
            s["frames"].append(torch.cat([f, torch.zeros((1, h, w), device=DEV)]).permute(1, 2, 0).to(dt).contiguous())
        s["out"] = torch.empty((h, w, 4), device=DEV)
        s["surf"] = registration.SURF(64, 64)
    else:
        (wl, raw, _), = _frames(dict(case, kind="frame", levels=5), seed)
        dt = torch.float16 if _half(case) else torch.float32
        p = _params(wl)
        s.update(conv=g.RawConverter(0), pattern=wl.pattern, scaled=_scaled(raw, p, torch.float32).to(dt).contiguous())
        _, _, s["ycc"], _ = _ycc_input(case, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        half = _half(case)
        return s["conv"].demosaic(s["raws"][0], s["params"][0], noiseReduction=True, fp16=half, out=s["outs"][0],
                                  out_fp16=half, postProcess=case["post"])
    if kind == "batch":
        return s["conv"].demosaic_batch(s["raws"], s["params"], s["outs"])
    if kind == "denoise":
        y, gr, o = s["views"]
        g.check(g.lib().gls_pyramid_denoise(s["conv"].handle, C.byref(y), C.byref(gr), C.byref(s["p"]),
                                            g.FP16_STORAGE if _half(case) else 0, C.byref(o), None))
        return s["out"]
    if kind == "calibrate":
        loss, grad = adjoint.loss_and_grad(s["conv"], s["raw"], s["p"], s["target"])
        return {"loss": np.array([loss]), "grad": grad}
    if kind == "detect":
        kps, desc = s["surf"].detectAndCompute(s["plane"], 0)
        return {"desc": desc, **{f: np.ascontiguousarray(kps[f]) for f in kps.dtype.names}}
    if kind == "register":
        n = case["n"]
        return s["surf"].register_frames([0, 1], [[2 * f, 2 * f + 1] for f in range(1, n)], 1.0, 2000, True)
    if kind == "fuse":
        return registration.fuse_pyramid(s["surf"], s["frames"], s["Hs"], s["out"], case["levels"],
                                         case["robustness"])
    return {"raw": np.stack(s["conv"].MeasureRawNLF(s["scaled"], s["pattern"])),
            "ycc": np.stack(s["conv"].MeasureYCbCrNLF(s["ycc"]))}


# ------------------------------------------------------------------ work
TAPS, TAP_FLOPS = 441, 44  # block matching: 8-term distance, two exponentials, five sums


def _pyramid_px(px, levels):
    return sum(px / 4 ** l for l in range(levels))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        px = sum(int(a) * int(b) for a, b in (s.split("x") for s in case["sizes"].split(",")))
    else:
        px = case["w"] * case["h"]
    es = 2 if _half(case) else 4
    if kind in ("frame", "batch"):  # raw in, RGBA out
        return {"bytes": px * (2 + 4 * es), "flops": _pyramid_px(px, case["levels"]) * TAPS * TAP_FLOPS + 500 * px}
    if kind == "denoise":  # YCbCr and gradient in, YCbCr out
        return {"bytes": px * 10 * es, "flops": _pyramid_px(px, case["levels"]) * TAPS * TAP_FLOPS}
    if kind == "calibrate":  # raw and target in; the weights forward, then both sides of each pair backward
        return {"bytes": px * (2 + 12), "flops": _pyramid_px(px, case["levels"]) * TAPS * (TAP_FLOPS + 90)}
    if kind == "detect":  # 4 octaves x 4 layers of box filters
        return {"bytes": px * 4 + case["features"] * 284, "flops": px * 4 * 60 * (1 + 1 / 4 + 1 / 16 + 1 / 64)}
    if kind == "register":  # brute-force matching, then 2000 hypotheses (Jacobi, FP64) per pair
        jobs, k = 2 * (case["n"] - 1), case["features"]
        return {"bytes": (jobs + 2) * k * 284, "flops": jobs * (k * k * 192 + 2000 * (30 * 200 + k * 20))}
    if kind == "fuse":  # the frames in, RGBA out
        return {"bytes": px * (case["n"] * 4 * es + 16), "flops": px * case["n"] * 4 / 3 * 80}
    return {"bytes": px * 5 * es, "flops": px * (81 * 2 + 25 * 6)}  # the two planes in


# ------------------------------------------------------------------ float64
def _matrices(p):
    """cam -> YCbCr and its inverse, 3 x 3 lists."""
    rc, xyz = np.array(p.rgb_cam[:]).reshape(3, 3), np.array(p.xyz_rgb[:])
    kr, kg, kb = xyz[3:6] @ rc
    m = np.array([[kr, kg, kb], [-0.5 * kr / (1 - kb), -0.5 * kg / (1 - kb), 0.5],
                  [0.5, -0.5 * kg / (1 - kr), -0.5 * kb / (1 - kr)]])
    return m.tolist(), np.linalg.inv(m).tolist()


def _pad(t, r):
    """t (h, w) with r clamped rows and columns around."""
    return F.pad(t[None, None], (r, r, r, r), mode="replicate")[0, 0]


def _sstep(a, b, x):
    t = ((x - a) / (b - a)).clamp(0, 1)
    return t * t * (3 - 2 * t)


def _mix(a, b, t):
    return a + (b - a) * t


def _scaled(raw, p, dtype):
    """scaleRawData: 0.1 + 0.9 (raw - black) / range, not below 0 (equal gains)."""
    v = (raw.to(torch.int32) & 0xffff).to(dtype) - round(p.black_level)
    return (v * (p.scale_mul[0] * 0.9 / 65535.0) + 0.1).clamp(min=0)


def _gradient(s, v0, v1):
    """Sobel of the raw plane, Gaussian-blurred: narrow where it stands out
    of the noise, wide elsewhere; |g| blurred, with the signs of blurred g."""
    h, w = s.shape
    q = _pad(s, 1)
    t = lambda dx, dy: q[1 + dy:1 + dy + h, 1 + dx:1 + dx + w]  # noqa: E731
    gx = (t(-1, -1) - t(1, -1) + 2 * (t(-1, 0) - t(1, 0)) + t(-1, 1) - t(1, 1)) / math.sqrt(4.5)
    gy = (t(-1, -1) - t(-1, 1) + 2 * (t(0, -1) - t(0, 1)) + t(1, -1) - t(1, 1)) / math.sqrt(4.5)

    def blur(radius):
        ks = max(math.ceil(2 * radius), 2) | 1
        r = ks // 2
        k = [math.exp(-(i * i) / (2 * radius * radius)) for i in range(-r, r + 1)]
        out = []
        for c in (gx, gy, gx.abs(), gy.abs()):
            P = _pad(c, r + 1)
            at = lambda dx, dy: P[r + 1 + dy:r + 1 + dy + h, r + 1 + dx:r + 1 + dx + w]  # noqa: E731
            rows = sum(k[i + r] * P[:, r + 1 + i:r + 1 + i + w] for i in range(-r, r + 1))
            acc = sum(k[j + r] * rows[r + 1 + j:r + 1 + j + h] for j in range(-r, r + 1))
            # the last corner tap is read half a pixel further out
            corner = (at(r, r) + at(r + 1, r) + at(r, r + 1) + at(r + 1, r + 1)) / 4
            out.append((acc + k[-1] * k[-1] * (corner - at(r, r))) / sum(k) ** 2)
        return out

    a, b = blur(1.5), blur(4.5)
    wide = torch.hypot(a[0], a[1]) < 4 * (v0 + v1 * s).sqrt()
    n = [torch.where(wide, y, x) for x, y in zip(a, b)]
    return torch.copysign(n[2], n[0]), torch.copysign(n[3], n[1])


OFFS = ((0, 0), (0, 1), (1, 1), (1, 0))  # RGGB: (x, y) of R, G, B, G2


def _quads(s):
    return [s[oy::2, ox::2] for ox, oy in OFFS]


def _nine(t):
    h, w = t.shape
    P = _pad(t, 1)
    return torch.stack([P[1 + j:1 + j + h, 1 + i:1 + i + w] for j in (-1, 0, 1) for i in (-1, 0, 1)]).sort(0)[0]


def _raw_denoise(s, gx, gy, var, strength):
    """The high-noise branch: despeckle, then 5 x 5 cross-channel denoise of the quads."""
    mag = torch.hypot(gx[0::2, 0::2], gy[0::2, 0::2])
    q = []
    for c, v in enumerate(_quads(s)):
        n = _nine(v)
        sg = (var[c] * v).sqrt()
        tex = 1 - 0.5 * _sstep(1.0, 2.0, mag / sg)
        mn = _mix(n[0], n[1], tex * (1 - _sstep(2 * sg, 8 * sg, n[1] - n[0])))
        mx = _mix(n[8], n[7], tex * (1 - _sstep(sg, 4 * sg, n[8] - n[7])))
        q.append(torch.minimum(torch.maximum(v, mn), mx))
    inv = [1 / (strength * (var[c] * (q[c] + 0.0001)).sqrt()) for c in range(4)]
    P = [_pad(v, 2) for v in q]
    h, w = q[0].shape
    tot, sums = 0, [0, 0, 0, 0]
    for j in range(5):
        for i in range(5):
            t = [v[j:j + h, i:i + w] for v in P]
            wt = torch.exp(-2 * sum(((q[c] - t[c]) * inv[c]) ** 2 for c in range(4)))
            tot = tot + wt
            sums = [a + wt * b for a, b in zip(sums, t)]
    out = torch.zeros_like(s)
    for c, (ox, oy) in enumerate(OFFS):
        out[oy::2, ox::2] = sums[c] / tot
    return out


def _demosaic(s, gx, gy, rv, gv, bv):
    """Green, red/blue at blue/red, red/blue at green, highlights: camera RGB."""
    h, w = s.shape
    y, x = torch.meshgrid(torch.arange(h, device=s.device) & 1, torch.arange(w, device=s.device) & 1, indexing="ij")
    red, blue = (x == 0) & (y == 0), (x == 1) & (y == 1)
    rb = red | blue

    def reader(t, r):
        P = _pad(t, r)
        return lambda dx, dy: P[r + dy:r + dy + h, r + dx:r + dx + w]

    gx, gy = gx.abs(), gy.abs()
    glen, ang = torch.hypot(gx, gy), 2 * torch.atan2(gy, gx) / math.pi
    R = reader(s, 2)
    mx = lambda *v: torch.stack(v).amax(0)  # noqa: E731
    mn = lambda *v: torch.stack(v).amin(0)  # noqa: E731
    cl, cr, cu, cd = R(-2, 0), R(2, 0), R(0, -2), R(0, 2)
    gl, gr, gu, gd = R(-1, 0), R(1, 0), R(0, -1), R(0, 1)
    diag = (R(-1, -1) + R(1, -1) + R(-1, 1) + R(1, 1)) / 4
    gave = (gl + gr + gu + gd) / 4
    low = 1 - _sstep(3.5e-4, 2e-3, torch.as_tensor(gv[1], dtype=s.dtype, device=s.device))
    sd = (gv[0] + gv[1] * gave).sqrt()
    sharp = (0.5 + 0.5 * low) * _sstep(sd, 4 * sd, glen) * (1 + low * (1 - _sstep(2 * sd, 8 * sd, glen)))
    hl = 1 - _sstep(0.25, 1.0, mx(s, cl, cr, cu, cd))
    d = ang
    if float(gv[1]) < 1e-3:
        d = torch.where(ang < 0.5, ang * _sstep(0.3, 0.45, ang), _mix(ang, 1.0, _sstep(0.55, 0.7, ang)))
    white = mn(s, gave, diag) / mx(s, gave, diag)
    k = hl * white * sharp
    gv_ = _mix((gu + gd) / 2 - k * ((cu + cd) - 2 * s) / 4, (gl + gr) / 2 - k * ((cl + cr) - 2 * s) / 4, d)
    gv_ = torch.minimum(torch.maximum(gv_, _mix(1.0, 0.5, white) * mn(gl, gr, gu, gd)),
                        _mix(1.0, 1.5, white) * mx(gl, gr, gu, gd))
    green = torch.where(rb, gv_, s)

    G = reader(green, 2)
    v0, v1 = torch.where(red, rv[0], bv[0]), torch.where(red, rv[1], bv[1])
    tl, tr, bl, br = R(-1, -1), R(1, -1), R(-1, 1), R(1, 1)
    sd = (v0 + v1 * diag).sqrt()
    alpha = _mix(0.5, 1 - ang, _sstep(sd, 4 * sd, glen))
    hl = 1 - _sstep(0.25, 1.0, mx(green, G(2, -2), G(-2, 2), G(-2, -2), G(2, 2)))
    gc = green - s
    cd_ = lambda dx, dy: G(dx, dy) - R(dx, dy)  # noqa: E731
    aa = (cd_(1, -1) + cd_(-1, 1)) / 2 + hl * (cd_(2, -2) + cd_(-2, 2) - 2 * gc) / 8
    bb = (cd_(-1, -1) + cd_(1, 1)) / 2 + hl * (cd_(-2, -2) + cd_(2, 2) - 2 * gc) / 8
    other = green - _mix(aa, bb, alpha)
    other = torch.minimum(torch.maximum(other, mn(tl, tr, bl, br)), mx(tl, tr, bl, br))
    zero = torch.zeros_like(s)
    tr_ = torch.where(red, s, torch.where(blue, other, zero))
    tb_ = torch.where(blue, s, torch.where(red, other, zero))

    G = reader(green, 3)

    def at_green(t, v):
        T = reader(t, 3)
        l, r, u, dn = T(-1, 0), T(1, 0), T(0, -1), T(0, 1)
        e = lambda dx, dy: G(dx, dy) - T(dx, dy)  # noqa: E731
        sd = (v[0] + v[1] * (l + r + u + dn) / 4).sqrt()
        al = _mix(0.5, ang, _sstep(sd, 4 * sd, glen))
        hl = 1 - _sstep(0.25, 1.0, mx(green, G(1, 0), G(-1, 0), G(0, 1), G(0, -1)))
        vert = (e(0, -1) + e(0, 1)) / 2 - hl * ((e(0, 3) - e(0, -1)) - (e(0, 1) - e(0, -3))) / 8
        horz = (e(-1, 0) + e(1, 0)) / 2 - hl * ((e(3, 0) - e(-1, 0)) - (e(1, 0) - e(-3, 0))) / 8
        o = green - _mix(vert, horz, al)
        return torch.minimum(torch.maximum(o, mn(l, r, u, dn)), mx(l, r, u, dn))

    r_, b_ = torch.where(rb, tr_, at_green(tr_, rv)), torch.where(rb, tb_, at_green(tb_, bv))
    # blendHighlights, clip 1
    over = (r_ > 1) | (green > 1) | (b_ > 1)
    s3 = math.sqrt(3.0)
    lab = lambda a, b, c: (s3 * a - s3 * b, -a - b + 2 * c)  # noqa: E731
    y0, z0 = lab(r_, green, b_)
    y1, z1 = lab(r_.clamp(max=1), green.clamp(max=1), b_.clamp(max=1))
    n0 = y0 * y0 + z0 * z0
    ok = over & (n0 > 0)
    chroma = torch.where(ok, ((y1 * y1 + z1 * z1) / torch.where(ok, n0, 1.0) + 1e-300).sqrt(), 1.0)
    x0, yy, zz = r_ + green + b_, y0 * chroma, z0 * chroma
    pick = lambda v, o: torch.where(over, v / 3, o)  # noqa: E731
    return torch.stack([pick(x0 + s3 / 2 * yy - 0.5 * zz, r_), pick(x0 - s3 / 2 * yy - 0.5 * zz, green),
                        pick(x0 + zz, b_)])


def _despeckle(ycc, va, vb):
    n = _nine(ycc[0])
    sg = (va + vb * ycc[0]).sqrt()
    mn = _mix(n[1], n[0], _sstep(sg, 4 * sg, n[1] - n[0]))
    mx = _mix(n[7], n[8], _sstep(sg, 4 * sg, n[8] - n[7]))
    return torch.stack([torch.minimum(torch.maximum(ycc[0], mn), mx), _nine(ycc[1])[4], _nine(ycc[2])[4]])


def _sample(img, u, v):
    """img (c, h, w) at texel positions v x u, bilinear, clamped."""
    h, w = img.shape[-2:]
    fu, fv = u.floor(), v.floor()
    ax, ay = u - fu, (v - fv)[:, None]
    xi, yi = fu.long(), fv.long()
    rows = [img[:, (yi + k).clamp(0, h - 1)] for k in (0, 1)]
    top, bot = ((1 - ax) * r[..., xi.clamp(0, w - 1)] + ax * r[..., (xi + 1).clamp(0, w - 1)] for r in rows)
    return (1 - ay) * top + ay * bot


def _down(img, ow, oh):
    h, w = img.shape[-2:]
    x, y = torch.arange(ow, device=DEV, dtype=F64), torch.arange(oh, device=DEV, dtype=F64)
    return sum(_sample(img, (x + a) * (w / ow) - 0.5, (y + b) * (h / oh) - 0.5) for a in (0, 1) for b in (0, 1)) / 4


def _up(img, w, h):
    cw, ch = img.shape[-1], img.shape[-2]
    return _sample(img, (torch.arange(w, device=DEV, dtype=F64) + 0.5) * (cw / w) - 0.5,
                   (torch.arange(h, device=DEV, dtype=F64) + 0.5) * (ch / h) - 0.5)


def _pca(y):
    """The 8 leading components (25, 8) of the 5 x 5 patches at every eighth pixel."""
    h, w = y.shape
    P = _pad(y, 2)
    v = torch.stack([P[j:j + 8 * (h // 8):8, i:i + 8 * (w // 8):8].reshape(-1) for j in range(5) for i in range(5)], 1)
    v = v - v.mean(0)
    return torch.linalg.eigh(v.T @ v / (v.shape[0] - 1))[1][:, -8:].flip(1)


def _window_row(j, layer, pca, L, k1, k2):
    h, w = L.shape
    lp, pp = F.pad(layer[None], (10,) * 4, mode="replicate")[0], F.pad(pca[None], (10,) * 4, mode="replicate")[0]
    sums = [0, 0, 0, 0, 0]
    for i in range(21):
        q = lp[:, j:j + h, i:i + w]
        d2 = ((pp[:, j:j + h, i:i + w] - pca) ** 2).sum(0)
        lw = torch.exp(-2 * d2 * L * L)
        cw = torch.exp(-2 * (lw * lw + ((q[1] - layer[1]) * k1) ** 2 + ((q[2] - layer[2]) * k2) ** 2))
        sw = math.exp(-0.02 * ((i - 10) ** 2 + (j - 10) ** 2))
        for n, t in enumerate((sw * lw * q[0], sw * cw * q[1], sw * cw * q[2], sw * lw, sw * cw)):
            sums[n] = sums[n] + t
    return sums


def _denoise(ycc, gx, gy, p, theta=None):
    """The pyramid denoise: (Y, Cb, Cr, sum of luma weights), (4, h, w). theta:
    the calibration vector (luma, chroma, A_Y, B_Y, A_C, B_C by level) to
    differentiate, in the place of the parameters' values; bases held fixed."""
    n = p.levels
    img, grad = [ycc], [torch.stack([gx, gy])]
    h, w = ycc.shape[-2:]
    for l in range(1, n):
        img.append(_down(img[-1], w >> l, h >> l))
        grad.append(_down(grad[-1], w >> l, h >> l))
    den = None
    for l in range(n - 1, -1, -1):
        d, nl = p.denoise[l], p.pyramid_nlf[l]
        luma, chroma, a, b = d.luma, d.chroma, list(nl.a), list(nl.b)
        if theta is not None:
            luma, chroma = theta[l], theta[5 + l]
            a = [theta[10 + l], theta[20 + l], theta[20 + l] + (a[2] - a[1])]
            b = [theta[15 + l], theta[25 + l], theta[25 + l] + (b[2] - b[1])]
        layer, mag = img[l], torch.hypot(grad[l][0], grad[l][1])
        if l < n - 1:
            u, v = _up(img[l + 1], w >> l, h >> l), _up(den[:3], w >> l, h >> l)
            alpha = d.sharpening
            if alpha > 1:
                sg = (a[0] * luma + b[0] * luma * v[0]).sqrt()
                alpha = 1 + (alpha - 1) * (_sstep(sg, 4 * sg, mag) * (1 - _sstep(0.75, 0.95, v[0])) *
                                           _sstep(0.05, 0.1, v[0]))
            layer = v + (img[l] - (u - v) - v) * alpha
            layer = torch.cat([layer[:1].clamp(min=0), layer[1:]])
        basis = _pca(layer[0].detach())
        P = _pad(layer[0], 2)
        hl, wl = layer.shape[-2:]
        pca = sum(P[j:j + hl, i:i + wl] * basis[5 * j + i][:, None, None] for j in range(5) for i in range(5))
        sg = [(a[c] + b[c] * layer[0]).sqrt() for c in range(3)]
        L = 1 / (luma * sg[0]) / (1 + d.gradient_boost * _sstep(2.0, 16.0, d.gradient_threshold * mag / sg[0]))
        k1, k2 = (1 / (chroma * sg[c]) / d.chroma_boost for c in (1, 2))
        sums = [0] * 5
        for j in range(21):
            if theta is None:
                row = _window_row(j, layer, pca, L, k1, k2)
            else:
                row = torch.utils.checkpoint.checkpoint(_window_row, j, layer, pca, L, k1, k2, use_reentrant=False)
            sums = [x + y for x, y in zip(sums, row)]
        den = torch.stack([sums[0] / sums[3], sums[1] / sums[4], sums[2] / sums[4], sums[3]])
    return den


def _rgb(raw, p, theta=None):
    """raw -> denoised camera RGB (3, h, w)."""
    nl = p.raw_nlf
    a, b = list(nl.a), list(nl.b)
    gv = [(a[1] + a[3]) / 2, (b[1] + b[3]) / 2]
    s = _scaled(raw, p, F64)
    gx, gy = _gradient(s, *gv)
    if theta is not None:  # the two raw green entries move G and G2 together
        gv = [theta[30], theta[31]]
        b[1], b[3] = b[1] + (theta[31] - (b[1] + b[3]) / 2), b[3] + (theta[31] - (b[1] + b[3]) / 2)
    if p.high_noise_image:
        s = _raw_denoise(s, gx, gy, b, p.raw_denoise_strength)
    cam = _demosaic(s, gx, gy, (a[0], b[0]), gv, (a[2], b[2]))
    fwd, inv = (torch.tensor(m, device=DEV, dtype=F64) for m in _matrices(p))
    ycc = torch.einsum("ij,jhw->ihw", fwd, cam)
    ycc = _despeckle(ycc, p.pyramid_nlf[0].a[0], p.pyramid_nlf[0].b[0])
    return torch.einsum("ij,jhw->ihw", inv, _denoise(ycc, gx, gy, p, theta)[:3])


def _with_w(t):
    return torch.cat([t, torch.zeros_like(t[:1])]).permute(1, 2, 0)


def _fused(case, s):
    """The weighted Laplacian-pyramid mean of the warped frames."""
    w, h, n = case["w"], case["h"], case["levels"]
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=F64), torch.arange(w, device=DEV, dtype=F64),
                          indexing="ij")
    acc, ref = [None] * n, None
    for f, img in enumerate(s["frames"]):
        t = img[..., :3].to(F64).permute(2, 0, 1)
        if f:
            H = np.asarray(s["Hs"][f], np.float64)
            d = H[2, 0] * x + H[2, 1] * y + H[2, 2]
            u = ((H[0, 0] * x + H[0, 1] * y + H[0, 2]) / d).clamp(-1, w)
            v = ((H[1, 0] * x + H[1, 1] * y + H[1, 2]) / d).clamp(-1, h)
            xi, yi = u.floor().long(), v.floor().long()
            ax, ay = u - xi, v - yi
            px = lambda i, j: t[:, (yi + j).clamp(0, h - 1), (xi + i).clamp(0, w - 1)]  # noqa: B023, E731
            t = _mix(_mix(px(0, 0), px(1, 0), ax), _mix(px(0, 1), px(1, 1), ax), ay)
        bands = []
        for l in range(n):
            c = _down(t, w >> (l + 1), h >> (l + 1)) if l + 1 < n else None
            bands.append(t - _up(c, w >> l, h >> l) if c is not None else t)
            t = c
        ref = ref or bands
        for l, b in enumerate(bands):
            wt = torch.exp(-case["robustness"] * ((b - ref[l]) ** 2).sum(0))
            acc[l] = (wt * b, wt) if f == 0 else (acc[l][0] + wt * b, acc[l][1] + wt)
    out = None
    for l in range(n - 1, -1, -1):
        b = acc[l][0] / acc[l][1]
        out = b if out is None else b + _up(out, w >> l, h >> l)
    return _with_w(out)


def _fit(m, v, pixels, raw):
    """The two-pass noise fit of (channels, positions) means and variances."""
    ok = (~v.isnan()).all(0) & (v[0] >= 0) if raw else (v > 0).all(0)
    top = v[:, ok].amax(0)
    hist = [int(((top > lo) & (top <= hi)).sum()) for lo, hi in
            ((-1, 1e-6), (1e-6, 1e-5), (1e-5, 1e-4), (1e-4, 1e-3), (1e-3, 1e-2))]
    bound = next((b for k, b in zip(hist, (1e-5, 1e-4, 1e-3, 1e-2, 1e-1)) if k > 1000), 1.0)

    def line(u):
        n = float(u.sum())
        sx, sy = m[:, u].sum(1), v[:, u].sum(1)
        sxx, sxy = (m[:, u] ** 2).sum(1), (m[:, u] * v[:, u]).sum(1)
        B = ((n * sxy - sx * sy) / (n * sxx - sx * sx)).clamp(min=1e-8)
        return ((sy - B * sx) / n).clamp(min=1e-8), B, n

    inside = ((m >= 0.001) & (m <= 0.9)).all(0)
    use = inside & (v <= bound).all(0)
    A, B, n = line(use)
    e2 = (A[:, None] + B[:, None] * m - v) ** 2
    use = inside & (v <= B[:, None]).all(0)  # the residuals and the second fit take variances under the slope
    err = torch.where((inside & (v <= bound).all(0)), e2, 0.0).sum(1) / n
    use = use & (e2 <= (0.5 if raw else 1.0) * err[:, None]).all(0)
    A2, B2, n2 = line(use)
    new = e2[:, use].sum(1) / n2
    better = bool((new < err).all() if raw else (new <= err).all())
    if better and n2 > (0.001 if raw else 0.01) * pixels:
        A, B = A2, B2
    return torch.stack([A, B])


def _box(t, r):
    P = _pad(t, r)
    h, w = t.shape
    rows = sum(P[:, i:i + w] for i in range(2 * r + 1))
    return sum(rows[j:j + h] for j in range(2 * r + 1))


def _noise_models(s):
    t = s["scaled"].to(F64)
    h, w = t.shape
    s1, s2 = _box(t, 4), _box(t * t, 4)
    var = (s2 - s1 * s1 / 81) / 81
    pick = lambda v: torch.stack([q.reshape(-1) for q in _quads(v)])  # noqa: E731
    raw = _fit(pick(s1 / 81), pick(var), w * h, True)
    c = s["ycc"].to(F64).permute(2, 0, 1)
    v = torch.stack([((_box(x * x, 2) - _box(x, 2) ** 2 / 25) / 25).reshape(-1) for x in c[:3]])
    m = (_box(c[0], 2) / 25).reshape(1, -1).expand(3, -1)
    return {"raw": raw, "ycc": _fit(m, v, c[0].numel(), False)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        if case["post"]:  # histogram bins and seeded film grain: held to the bound of its type
            return None
        (wl, raw, _), = _frames(case, seed)
        return _with_w(_rgb(raw, _params(wl)))
    if kind == "batch":
        return [_with_w(_rgb(raw, _params(wl))) for wl, raw, _ in _frames(case, seed)]
    if kind == "denoise":
        _, p, ycc, grad = _ycc_input(case, seed)
        c, d = ycc.to(F64).permute(2, 0, 1), grad.to(F64).permute(2, 0, 1)
        return _denoise(c[:3], d[0], d[1], p).permute(1, 2, 0)
    if kind == "calibrate":
        (wl, raw, rgb), = _frames(case, seed)
        p = _params(wl)
        theta = torch.tensor(adjoint.params_to_theta(p), device=DEV, dtype=F64, requires_grad=True)
        loss = ((_rgb(raw, p, theta) - (0.1 + 0.9 * rgb.to(torch.float32)).to(F64)) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach().reshape(1), "grad": theta.grad}
    if kind in ("detect", "register"):
        # keypoints, matches and models are chosen by comparisons of FP32
        # values in a fixed operation order: float64 chooses others
        return None
    s = prepare(case, seed)
    return _fused(case, s) if kind == "fuse" else _noise_models(s)
