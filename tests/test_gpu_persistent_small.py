"""The persistent batch with levels too small for a PCA patch, which have no
covariance task between the reconstruct tiles and block matching."""
import numpy as np
import pytest
import torch

from glasscamerapublic_b200 import scene

pytestmark = pytest.mark.gpu

SIZES = [(202, 48), (48, 72), (416, 58), (38, 36), (100, 44), (72, 34)]


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_levels_without_patches_match_the_stream_batch(converter, seed):
    raws, params = [], []
    for k, (w, h) in enumerate(SIZES * 2):
        wl = scene.Workload("p", w, h, levels=5, gain=1.0, read=3.0, iso=800, seed=100 * seed + k)
        raws.append(torch.from_numpy(scene.make_raw(wl)[0].view(np.int16)).cuda())
        params.append(scene.make_params(wl))
    ref, got = ([torch.empty((h, w, 4), dtype=torch.float16, device="cuda") for w, h in SIZES * 2] for _ in range(2))
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    converter.demosaic_batch(raws, params, ref, stream=st)
    converter.demosaic_batch(raws, params, got, stream=st, persistent=True)
    st.synchronize()
    for a, b in zip(ref, got):
        assert torch.equal(a, b)
