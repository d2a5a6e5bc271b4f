"""The device eigen-solve of the patch covariance against float64 numpy, over
spectra that take its different branches: separated and clustered
eigenvalues, rank-deficient patch sets, flat images, extreme scales."""
import ctypes as C

import numpy as np
import pytest

import glasscamerapublic_b200 as g

pytestmark = pytest.mark.gpu


def _basis(luma):
    import torch
    h, w = luma.shape
    img = torch.zeros((h, w, 4), device="cuda")
    img[..., 0] = torch.from_numpy(luma).cuda()
    out = torch.zeros((25, 8), device="cuda")
    v = g.ImageView(C.c_void_p(img.data_ptr()), w, h, 4, g.F32, w * 16)
    g.check(g.lib().gls_pca_basis_noalloc(C.byref(v), C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    return out.cpu().numpy().astype(np.float64)


def _covariance(luma):
    h, w = luma.shape
    P = np.pad(luma.astype(np.float64), 2, mode="edge")
    v = np.stack([P[j:j + 8 * (h // 8):8, i:i + 8 * (w // 8):8].reshape(-1) for j in range(5) for i in range(5)], 1)
    return np.cov(v.T)


def _image(kind, h, w):
    rng = np.random.default_rng(len(kind) * 1000 + h)
    y, x = np.mgrid[0:h, 0:w]
    if kind == "scene":
        a = 0.3 + 0.1 * np.sin(x / 9.0) + 0.1 * np.cos(y / 7.0) + 0.01 * rng.standard_normal((h, w))
    elif kind == "noise":  # all eigenvalues close
        a = 0.5 + 0.01 * rng.standard_normal((h, w))
    elif kind == "impulses":
        a = (rng.random((h, w)) < 0.02) * 1.0
    elif kind == "tiny":  # variances near 1e-13
        a = 1e-3 + 3e-7 * rng.standard_normal((h, w))
    elif kind == "huge":
        a = 1e4 * rng.standard_normal((h, w))
    else:  # equal pairs: patches that are single pixels of random sign, four positions alike
        a = np.zeros((h, w))
        for k, (dy, dx) in enumerate([(0, 0), (0, 1), (1, 0), (1, 1), (-1, 0), (0, -1), (-1, -1), (2, 2), (1, -1)]):
            gy, gx = np.mgrid[0:h // 8, 0:w // 8]
            on = (gy * (w // 8) + gx) % 9 == k
            yy, xx = 8 * gy[on] + dy, 8 * gx[on] + dx
            ok = (yy >= 0) & (xx >= 0)
            a[yy[ok], xx[ok]] = 1.0
    return a.astype(np.float32)


@pytest.mark.parametrize("kind", ["scene", "noise", "impulses", "tiny", "huge", "pairs"])
@pytest.mark.parametrize("h,w", [(72, 72), (40, 48), (264, 264)])
def test_basis_spans_the_leading_eigenspace(kind, h, w):
    img = _image(kind, h, w)
    b, c = _basis(img), _covariance(img)
    lam, V = np.linalg.eigh(c)
    lam, V = lam[::-1], V[:, ::-1]
    # FP32 rounding of the entries: 8 products of two roundings of 2^-25 each
    assert np.abs(b.T @ b - np.eye(8)).max() < 1e-6
    k = min(8, int((lam > 1e-8 * lam[0]).sum()))
    # the captured variance is the largest possible, to rounding
    got = np.array([b[:, i] @ c @ b[:, i] for i in range(k)])
    assert np.abs(got - lam[:k]).max() < 1e-6 * lam[0]
    # where the space is separated from the rest, the projectors agree
    gap = (lam[k - 1] - (lam[k] if k < 25 else 0.0)) / lam[0]
    if gap > 1e-4:
        assert np.abs(b[:, :k] @ b[:, :k].T - V[:, :k] @ V[:, :k].T).max() < 1e-6
    # signed so that the largest entry of a column is positive
    assert all(b[np.abs(b[:, i]).argmax(), i] > 0 for i in range(8))


@pytest.mark.parametrize("h,w", [(16, 16), (16, 24), (8, 24)])  # 4, 6 and 3 patches: rank 3, 5 and 2
def test_rank_deficient_basis_is_completed_as_on_the_host(h, w):
    from glasscamerapublic_b200 import scene
    rng = np.random.default_rng(h * w)
    ycc = np.zeros((h, w, 4), np.float32)
    ycc[..., 0] = rng.random((h, w))
    p = scene.make_params(scene.Workload("t", w, h, levels=1))
    conv = g.RawConverter(0)
    try:
        grad = np.zeros((h, w, 2), np.float32)
        g.PyramidProcessor(conv).denoise(ycc, grad, p)
        dev = conv.pca_basis(0).astype(np.float64)
        g.PyramidProcessor(conv).denoise(ycc, grad, p, host_pca=True)
        host = conv.pca_basis(0).astype(np.float64)
    finally:
        conv.close()
    assert np.abs(dev - host).max() < 1e-5


def test_flat_image_gives_the_unit_basis():
    b = _basis(np.full((64, 64), 0.25, np.float32))
    assert np.array_equal(b, np.eye(25, 8))
