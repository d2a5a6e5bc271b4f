"""The FP16 path's separable gradient blur against the FP32 path's bilinear taps
at the edges of its tiles, each blur on its own."""
import numpy as np
import pytest

import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(32, 32), (34, 66), (40, 30), (100, 38), (140, 134)])
@pytest.mark.parametrize("variance", [0.0, 1.0])
def test_fp16_gradient_follows_the_fp32_one(w, h, variance):
    """Variance 0 takes the narrow blur everywhere, 1 the wide one. Half rounding
    moves a raw value below 1 by 2^-12, a Sobel value (weights of 8 in all, over
    sqrt(4.5)) by 9e-4, a blurred magnitude by no more, its own rounding by 2^-12."""
    wl = scene.Workload("t", w, h, levels=1, gain=0.8, read=3.0, iso=400, seed=w + h)
    raw, _ = scene.make_raw(wl)
    p = scene.make_params(wl)
    for c in range(4):
        p.raw_nlf.a[c], p.raw_nlf.b[c] = variance, 0.0
    planes = []
    conv = g.RawConverter(0)
    try:
        for half in (False, True):
            conv.demosaic(raw, p, fp16=half)
            planes.append(np.abs(conv.plane(g.PLANE_GRADIENT).astype(np.float32)))
    finally:
        conv.close()
    assert planes[0].max() > 0.02
    assert np.abs(planes[0] - planes[1]).max() < 1.3e-3
