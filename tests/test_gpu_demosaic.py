"""The FP16-storage path's demosaic on its own planes against the oracle's FP32
run on the same planes, where a gradient has overflowed the half."""
import numpy as np
import pytest

import _oracle as O
import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern", [0, 1, 2, 3])
def test_a_gradient_beyond_the_half_keeps_its_direction(pattern):
    """One blue site beyond 65504 makes the blurred gradient around it (inf, inf),
    whose direction is the diagonal's, 45 degrees. The green of the red and blue
    sites 3 to 5 away (radius of the stencil: 2) is then the mean of its two
    estimates. Bound: the half's rounding, and 20 FP32 operations on values below 2."""
    w = h = 96
    rng = np.random.default_rng(pattern)
    p = scene.make_params(scene.Workload("t", w, h, levels=1, gain=0.8, read=3.0, iso=400, pattern=pattern))
    off = {0: ((1, 0), (0, 1)), 1: ((0, 1), (1, 0)), 2: ((0, 0), (1, 1)), 3: ((1, 1), (0, 0))}[pattern]  # red, blue
    for c in range(4):  # channels R, G, B, G2; the wide blur everywhere
        p.scale_mul[c] = 1.2 * 65535 / 0.9 if c == 2 else 65535 / 0.9 / 4000
        p.raw_nlf.a[c], p.raw_nlf.b[c] = 4.0, 0.0
    p.black_level = 500.0
    raw = (500 + rng.integers(0, 3000, (h, w))).astype(np.uint16)
    bx, by = off[1]
    raw[by::2, bx::2] = 500
    hx, hy = bx + 48, by + 40
    raw[hy, hx] = 65535
    conv = g.RawConverter(0)
    try:
        conv.demosaic(raw, p, noiseReduction=False, fp16=True)
        s = conv.plane(g.PLANE_SCALED_RAW)[..., 0].astype(np.float32)
        gr = conv.plane(g.PLANE_GRADIENT).astype(np.float32)
        got = conv.plane(g.PLANE_DEMOSAIC)[..., 1].astype(np.float32)
    finally:
        conv.close()
    y, x = np.mgrid[0:h, 0:w]
    far = np.maximum(np.abs(x - hx), np.abs(y - hy))
    site = (far >= 3) & np.isinf(gr).all(-1)  # red and blue sites that see the overflow in the gradient alone
    site &= ((x & 1) == off[0][0]) & ((y & 1) == off[0][1]) | ((x & 1) == bx) & ((y & 1) == by)
    assert np.isinf(s[hy, hx]) and site.sum() >= 8
    ref = O.stage("demosaic_rgb", s, gr, p=p, w=w, h=h, out_shape=(h, w, 4), f64=False)[..., 1]
    assert np.isfinite(ref[site]).all()
    assert (np.abs(got - ref)[site] < ref[site] * 2.0 ** -11 + 20 * 2.0 ** -23).all()
