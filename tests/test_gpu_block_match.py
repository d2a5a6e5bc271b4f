"""The FP16 block matcher on its own (a one-level pyramid denoise) at the edges
of its tiles and at extreme values."""
import ctypes as C

import numpy as np
import pytest

import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import scene

pytestmark = pytest.mark.gpu


def _denoise(ycc, grad, p, fp16):
    import torch
    h, w = ycc.shape[:2]
    dt, code = (torch.float16, g.F16) if fp16 else (torch.float32, g.F32)
    t = [torch.from_numpy(a).cuda().to(dt).contiguous() for a in (ycc, grad)]
    out = torch.empty((h, w, 4), dtype=dt, device="cuda")
    v = [g.ImageView(C.c_void_p(a.data_ptr()), w, h, a.shape[2], code, a.stride(0) * a.element_size())
         for a in (t[0], t[1], out)]
    conv = g.RawConverter(0)
    try:
        g.check(g.lib().gls_pyramid_denoise(conv.handle, C.byref(v[0]), C.byref(v[1]), C.byref(p),
                                            (g.FP16_STORAGE if fp16 else 0) | g.SYNC, C.byref(v[2]), None))
        return out.float().cpu().numpy()
    finally:
        conv.close()


def _image(h, w, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    ycc = np.zeros((h, w, 4), np.float32)
    ycc[..., 0] = 0.4 + 0.2 * np.sin(x / 11.0) * np.cos(y / 7.0) + 0.01 * rng.standard_normal((h, w))
    ycc[..., 1:3] = 0.01 * rng.standard_normal((h, w, 2))
    grad = np.abs(0.01 * rng.standard_normal((h, w, 2))).astype(np.float32)
    return ycc.astype(np.float16).astype(np.float32), grad.astype(np.float16).astype(np.float32)


def _params(h, w, a=1e-5, b=1e-4, lsc=0.0):
    p = scene.make_params(scene.Workload("t", w, h, levels=1, iso=800))
    for c in range(3):
        p.pyramid_nlf[0].a[c], p.pyramid_nlf[0].b[c] = a, b
    p.lens_shading_correction = lsc
    return p


@pytest.mark.parametrize("h,w", [(1, 1), (3, 5), (16, 32), (17, 33), (15, 31), (33, 64), (70, 41), (4, 200), (200, 4)])
@pytest.mark.parametrize("lsc", [0.0, 0.5])
def test_fp16_matcher_follows_the_fp32_one(h, w, lsc):
    """Weights agree to the half-precision coefficients (2 |exponent| 2^-10, about
    3% where a weight counts), so a mean of deviations up to 4 sigma = 0.04
    moves by at most 1.2e-3, and half rounding adds 2.5e-4."""
    ycc, grad = _image(h, w, h * 1000 + w)
    p = _params(h, w, lsc=lsc)
    a, b = _denoise(ycc, grad, p, True), _denoise(ycc, grad, p, False)
    # the lens-shading radius of a 1 x 1 image is 0 / 0: undefined in both
    assert np.isfinite(b).all() or (h, w, lsc) == (1, 1, 0.5)
    ok = np.isfinite(b).all(-1)
    assert (np.abs(a[..., :3] - b[..., :3]) < 2e-3)[ok].all()
    assert (np.abs(a[..., 3] - b[..., 3]) < 0.05 * b[..., 3])[ok].all()


@pytest.mark.parametrize("h,w", [(64, 90), (128, 150), (192, 256), (250, 250), (303, 610)])
def test_fp16_tiles_split_over_blocks(h, w):
    """12, 40, 96, 128 and 380 tiles: their groups over 8, 4, 3, 2 and 1 blocks. Bounds as above."""
    ycc, grad = _image(h, w, h)
    p = _params(h, w)
    a, b = _denoise(ycc, grad, p, True), _denoise(ycc, grad, p, False)
    assert (np.abs(a[..., :3] - b[..., :3]) < 2e-3).all()
    assert (np.abs(a[..., 3] - b[..., 3]) < 0.05 * b[..., 3]).all()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_chroma_value_that_is_not_finite_stays_in_its_window(value):
    h, w, py, px = 75, 90, 44, 52
    ycc, grad = _image(h, w, 5)
    p = _params(h, w)
    clean = _denoise(ycc, grad, p, True)
    ycc[py, px, 1] = value
    got = _denoise(ycc, grad, p, True)
    y, x = np.mgrid[0:h, 0:w]
    outside = (np.abs(y - py) > 10) | (np.abs(x - px) > 10)
    # the same sums over the same taps, but for the constants of the one pixel
    assert np.array_equal(got[outside], clean[outside])
    assert np.array_equal(got[..., 0][outside], clean[..., 0][outside])


@pytest.mark.parametrize("var", [1e-14, 1e-30])
def test_extreme_distance_scales_keep_the_pixel(var):
    """Without noise nothing but identical patches is averaged."""
    h, w = 40, 70
    ycc, grad = _image(h, w, 6)
    got = _denoise(ycc, grad, _params(h, w, a=var, b=0.0), True)
    assert np.isfinite(got).all()
    assert np.abs(got[..., :3] - ycc[..., :3]).max() < 1e-3


@pytest.mark.parametrize("h,w", [(1, 1), (3, 5), (4, 32), (5, 33), (17, 31), (70, 41),
                                 (148, 128), (149, 128), (149, 129), (401, 803)])
def test_fp32_matcher_against_float64(h, w):
    """One and two pixels a thread (128 x 148 is the largest with one). The
    coefficients' rounding (25 terms of 0.5 in FP32, 5e-7) moves an exponent by
    4 d s^2 5e-7: 1e-3 of a weight at |d s| = 3 and s = 130, so a mean of
    deviations up to 0.04 by at most 4e-5."""
    import torch
    import _torch_pyramid as TP
    ycc, grad = _image(h, w, h * 1000 + w)
    p = _params(h, w)
    t = [torch.from_numpy(a).cuda() for a in (ycc, grad)]
    out = torch.empty((h, w, 4), device="cuda")
    v = [g.ImageView(C.c_void_p(a.data_ptr()), w, h, a.shape[2], g.F32, a.stride(0) * 4) for a in (*t, out)]
    conv = g.RawConverter(0)
    try:
        g.check(g.lib().gls_pyramid_denoise(conv.handle, C.byref(v[0]), C.byref(v[1]), C.byref(p), g.SYNC,
                                            C.byref(v[2]), None))
        basis = torch.from_numpy(conv.pca_basis(0)).cuda().double()
    finally:
        conv.close()
    layer, dp = t[0].double(), p.denoise[0]
    nlf = [torch.tensor([float(q) for q in x], dtype=torch.float64, device="cuda")
           for x in (p.pyramid_nlf[0].a, p.pyramid_nlf[0].b)]
    ref = TP.block_match(layer, t[1].double(), TP.pca_project(layer, basis), *nlf,
                         (dp.luma, dp.chroma, dp.chroma), dp).cpu().numpy()
    got = out.cpu().numpy()
    assert np.abs(got[..., :3] - ref[..., :3]).max() < 4e-5
    assert (np.abs(got[..., 3] - ref[..., 3]) < 1e-3 * ref[..., 3]).all()
