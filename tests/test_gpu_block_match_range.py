"""The FP16 block matcher over the half's range: coefficients near its largest
value, and a luma value that is not finite."""
import numpy as np
import pytest

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
