"""The noise statistics over the range of frame sizes, bit-exact to the oracle."""
import numpy as np
import pytest

import _oracle as O
import glasscamerapublic_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [
    (1, 1), (33, 9),
    (768, 288), (768, 289), (767, 296),     # 864 tiles of 32 x 8, 888: one position a thread, two
    (768, 584), (768, 585), (766, 599),     # 1752, 1776: two, four
    (1100, 700),
])
@pytest.mark.parametrize("half", [False, True])
def test_ycbcr_statistics_by_size(converter, w, h, half):
    import torch
    rng = np.random.default_rng(w * h)
    ycc = rng.standard_normal((h, w, 4)).astype(np.float16)
    t = torch.from_numpy(ycc).cuda()
    converter.MeasureYCbCrNLF(t if half else t.float(), 1.0)
    st = converter.plane(g.PLANE_NLF_STATS)
    assert np.array_equal(st, O.ycc_noise_stats(ycc.astype(np.float32)))


@pytest.mark.parametrize("w,h", [(2, 2), (130, 18), (640, 482), (1026, 770)])
def test_raw_statistics_by_size(converter, w, h):
    import torch
    rng = np.random.default_rng(w * h)
    raw = rng.random((h, w), dtype=np.float32)
    converter.MeasureRawNLF(torch.from_numpy(raw).cuda(), 2, 1.0)
    om, ov = O.raw_noise_stats(raw, 2)
    assert np.array_equal(converter.plane(g.PLANE_NLF_MEAN), om)
    assert np.array_equal(converter.plane(g.PLANE_NLF_VAR), ov)
