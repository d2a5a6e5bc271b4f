"""The FP32 block matcher where a pixel's chroma weights all lie near FP32's smallest numbers."""
import numpy as np
import pytest

from test_gpu_block_match import _denoise, _image, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(64, 96), (150, 128)])  # one and two pixels a thread
@pytest.mark.parametrize("var", [1e-19, 1e-20])
def test_chroma_weights_below_the_smallest_normal_number_count(h, w, var):
    """The chroma difference c v - c v0 of the pixel itself is the rounding of c v0, which
    at these variances leaves it a weight of 2^-q, the only one of its window. Down to
    2^-149 that weight exists (one bit at the end): the mean is the pixel's
    own chroma within 2^(q - 148) of its size."""
    ycc, grad = _image(h, w, 3)
    ycc[..., 1:3] = (0.3 * np.random.default_rng(1).standard_normal((h, w, 2))).astype(np.float16)
    p = _params(h, w, a=var, b=0.0)
    d, f = p.denoise[0], np.float32
    k = f(2) * f(1.4426950408889634)
    c = f(np.sqrt(k)) * ((f(1) / (f(d.chroma) * np.sqrt(f(p.pyramid_nlf[0].a[1])))) / f(d.chroma_boost))
    exact = np.float64(c) * ycc[..., 1:3].astype(np.float64)
    rest = exact - exact.astype(np.float32)
    q = float(k) + (rest ** 2).sum(-1)
    band = (q > 127) & (q < 135)
    assert band.sum() > 20
    got = _denoise(ycc, grad, p, False)[..., 1:3]
    assert np.isfinite(got[q < 135]).all()
    err = np.abs(got - ycc[..., 1:3]).max(-1)
    assert (err < 2.0 ** (np.minimum(q, 160) - 148) * (1 + np.abs(ycc[..., 1:3]).max(-1)))[band].all()
