"""Which tiles the DoG sweep takes (csrc/sweep.cu, find_form): wide frames of few rows, and of heights on both sides of a
full wave of either tile, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(9800, 8, 2), (10001, 30, 2), (4000, 40, 3), (2001, 112, 3)])
def test_gpu_dog_of_wide_frames(W, H, D):
    import hdog
    sig = (2.0, 1.5, 3.2, 2.4)
    norm = np.random.default_rng(W + H).normal(0, 1, (D, H, W)).astype(np.float32)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D, sigma_xy_small=sig[0], sigma_z_small=sig[1],
                                       sigma_xy_large=sig[2], sigma_z_large=sig[3])) as ctx:
        got = ctx.dog(torch.from_numpy(norm).cuda()).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), orc.dog(norm, *sig).view(np.uint32))
