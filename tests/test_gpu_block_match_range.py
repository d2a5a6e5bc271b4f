"""The FP16 block matcher over the half's range: coefficients near its largest
value, and a luma value that is not finite."""
import numpy as np
import pytest

import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import scene
from test_gpu_block_match import _denoise, _image, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [5000.0, 8000.0, 12000.0])
def test_coefficients_up_to_the_largest_half(step):
    """Two flat halves `step` apart with noise of sigma 100, cut at 4 sigma: the first
    coefficient differs by 5 step, 25000 to 60000, from one half to the other. Only a
    half's own pixels count in a mean, so it stays within 4 sigma of the level, and the
    pixel itself keeps the sum of weights at 1 or more."""
    h, w = 70, 90
    rng = np.random.default_rng(int(step))
    level = np.where(np.arange(w) < 41, 300.0, 300.0 + step)[None].repeat(h, 0)
    ycc = np.zeros((h, w, 4), np.float32)
    ycc[..., 0] = level + np.clip(100.0 * rng.standard_normal((h, w)), -300, 400)
    grad = np.zeros((h, w, 2), np.float32)
    got = _denoise(ycc, grad, _params(h, w, a=1e4, b=0.0), True)
    assert np.isfinite(got[..., :3]).all() and (got[..., 3] >= 0.99).all()
    assert np.abs(got[..., 0] - level).max() < 400 + 8  # and the half's spacing


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("py,px", [(16, 48), (14, 46), (18, 50), (19, 44), (47, 48)])
def test_a_luma_value_that_is_not_finite_reaches_twelve_positions(value, py, px):
    """The patches of the window's positions hold it. Around the centre of a 32 x 32
    region, (16, 48), it would enter the coefficients' common offset. No sampled
    patch holds it (columns 43 on of a 55-wide image), so the basis is the clean image's.
    Beyond its reach the matcher follows the FP32 one within 1.5e-3 (the bound of the
    comparison with it) as the clean run does."""
    h, w = 75, 55
    ycc, grad = _image(h, w, 7)
    p = _params(h, w)
    clean = _denoise(ycc, grad, p, True)
    ycc[py, px, 0] = value
    got = _denoise(ycc, grad, p, True)
    y, x = np.mgrid[0:h, 0:w]
    outside = (np.abs(y - py) > 12) | (np.abs(x - px) > 12)
    assert outside[(y // 32 == py // 32) & (x // 32 == px // 32)].any()
    assert np.abs(got[..., :3] - clean[..., :3])[outside].max() < 3e-3
    assert (np.abs(got[..., 3] - clean[..., 3])[outside] < 0.1 * clean[..., 3][outside]).all()


@pytest.mark.parametrize("n", [2, 3, 6, 7])
@pytest.mark.parametrize("w,h,levels", [(64, 48, 1), (256, 192, 3), (322, 250, 3)])
def test_a_batch_that_splits_its_tiles_less_gives_the_same_bits(n, w, h, levels):
    """24 to 96 tiles, over 8 to 1 blocks by the number of streams: a frame alone and in a batch."""
    torch = pytest.importorskip("torch")
    raws, ps = [], []
    for k in range(n):
        wl = scene.Workload("t", w, h, levels=levels, gain=0.8, read=3.0, iso=400, seed=k)
        raws.append(torch.from_numpy(scene.make_raw(wl)[0].view(np.int16)).cuda())
        ps.append(scene.make_params(wl))
    conv = g.RawConverter(0)
    try:
        one = [conv.demosaic(r, p, noiseReduction=True, fp16=True, out_fp16=True,
                             out=torch.empty((h, w, 4), dtype=torch.float16, device="cuda")).clone()
               for r, p in zip(raws, ps)]
        outs = [torch.empty((h, w, 4), dtype=torch.float16, device="cuda") for _ in raws]
        conv.demosaic_batch(raws, ps, outs)
        torch.cuda.synchronize()
    finally:
        conv.close()
    for a, b in zip(one, outs):
        assert torch.equal(a, b)
