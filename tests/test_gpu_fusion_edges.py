"""Fusion at the frames' far edges: a sample there takes the last texel alone,
whatever the texel before it holds."""
import numpy as np
import pytest
import torch

from glasscamerapublic_b200.registration import SURF, fuse_pyramid, register_image

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    s = SURF(64, 64, max_features=10)
    yield s
    s.close()


@pytest.mark.parametrize("value", [np.inf, np.nan, -3e4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("shift", [0, 9])
def test_the_last_texels_stand_alone(ctx, value, dtype, axis, shift):
    """The mean of a frame and one whose second to last column (row) is out of
    range, unmoved or moved by 9 texels; where the sample lies on or beyond the
    last column the mean is the exact one of the edge texels."""
    w, h = 45, 37
    rng = np.random.default_rng(11)
    ref, frm = (torch.from_numpy(rng.random((h, w, 4)).astype(np.float32)).to(dtype) for _ in range(2))
    bad = (slice(None), w - 2) if axis else (h - 2,)
    ref[bad], frm[bad] = value, value
    H = np.eye(3, dtype=np.float32)
    H[0, 2], H[1, 2] = (shift, 0) if axis else (0, shift)
    out = torch.empty((h, w, 4), device="cuda")
    fuse_pyramid(ctx, [ref.cuda(), frm.cuda()], [np.eye(3, dtype=np.float32), H], out, levels=1, robustness=0.0)
    torch.cuda.synchronize()
    got = out.cpu().numpy()[..., :3]
    r, f = ref.float().numpy()[..., :3], frm.float().numpy()[..., :3]
    if axis:
        assert np.array_equal(got[:, w - 1], (r[:, w - 1] + f[:, w - 1]) / 2)
        for x in range(w - 1 - shift, w - 3):
            # the reference between two of its own texels: a + 0 (b - a)
            assert np.array_equal(got[:, x], (r[:, x] + f[:, w - 1]) / 2)
    else:
        assert np.array_equal(got[h - 1], (r[h - 1] + f[h - 1]) / 2)
        for y in range(h - 1 - shift, h - 3):
            assert np.array_equal(got[y], (r[y] + f[h - 1]) / 2)


@pytest.mark.parametrize("formats", ["f32", "f16", "mixed"])
@pytest.mark.parametrize("n,w,h,levels,sizes", [
    (2, 140, 17, 5, [(318, 9)]),
    (5, 129, 97, 3, []),
    (9, 96, 64, 2, [(96, 64), (1, 12), (45, 32)]),  # a group of the reference and one frame
])
def test_bursts_under_perspective(ctx, formats, n, w, h, levels, sizes):
    """Frames of every format and size under homographies with a perspective part,
    through the pyramid, against the float64 restatement on registerImage's
    warps. Positions agree to an ulp (2^-17 at 128 texels, slope up to 1), which the
    bands pass on at most twice over: within the restatement's 1e-4."""
    from test_gpu_fusion import _numpy_fusion
    rng = np.random.default_rng(n)
    frames, Hs = [], []
    for f in range(n):
        fw, fh = (w, h) if f == 0 or f > len(sizes) else sizes[f - 1]
        img = rng.random((fh, fw, 4), dtype=np.float32)
        half = formats == "f16" or (formats == "mixed" and f % 2 == 1)
        frames.append(img.astype(np.float16).astype(np.float32) if half else img)
        H = np.eye(3) + rng.standard_normal((3, 3)) * [[.02, .02, 5], [.02, .02, 5], [1e-4, 1e-4, 0]]
        Hs.append((np.eye(3) if f == 0 else H).astype(np.float32))
    warped = []
    for img, H in zip(frames, Hs):
        o = torch.empty((h, w, 4), device="cuda")
        register_image(torch.from_numpy(img).cuda(), o, H)
        warped.append(o.cpu().numpy().astype(np.float64))
    ref = _numpy_fusion(warped, levels, 20.0)
    t = [torch.from_numpy(img).cuda() for img in frames]
    if formats != "f32":
        t = [x.half() if formats == "f16" or f % 2 == 1 else x for f, x in enumerate(t)]
    out = torch.empty((h, w, 4), device="cuda")
    fuse_pyramid(ctx, t, Hs, out, levels=levels, robustness=20.0)
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy()[..., :3] - ref).max() < 1e-4
