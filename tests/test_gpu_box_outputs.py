"""The y box means (csrc/norm.cu, k_box_y) at each of their outputs per thread: 12 below 8 M voxels, 16 from there on,
20 for reaches from 64, with rows left over, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,r", [(97, 131, 3, 6), (97, 131, 3, 70), (40, 9, 2, 30), (521, 259, 63, 5), (1031, 1303, 7, 64)])
def test_gpu_box_means_along_y(W, H, D, r):
    import hdog
    v = np.random.default_rng(W + r).integers(0, 65536, (D, H, W)).astype(np.uint16)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=r, radius_norm_z=1, min_intensity=50,
                                       sigma_z_small=0.1, sigma_z_large=0.2, extra_depth_margin=0)) as ctx:
        norm = ctx.normalize(torch.from_numpy(v).cuda()).cpu().numpy()
    assert np.array_equal(norm.view(np.uint32), orc.normalize(v, r, 1, 50.0).view(np.uint32))
