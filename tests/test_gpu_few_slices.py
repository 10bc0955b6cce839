"""The z window pass (csrc/norm.cu, mm_z) on volumes of few slices, around the line between its two forms, for both
borders and every column width, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(40, 12), (42, 11), (41, 11)])      # slices on 8, 4 and 2 bytes
@pytest.mark.parametrize("rz", [1, 2, 5, 8])
@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 6])
def test_gpu_few_slices(W, H, D, rz):
    import hdog
    v = np.random.default_rng(W + 10 * D + rz).integers(0, 65536, (D, H, W)).astype(np.uint16)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=3, radius_norm_z=rz, min_intensity=50,
                                       sigma_z_small=0.1, sigma_z_large=0.2, extra_depth_margin=0)) as ctx:
        d = torch.from_numpy(v).cuda()
        norm, ero = ctx.normalize(d).cpu().numpy(), ctx.erosion(d, 2, rz).cpu().numpy()
    assert np.array_equal(norm.view(np.uint32), orc.normalize(v, 3, rz, 50.0).view(np.uint32))
    assert np.array_equal(ero, orc.erosion(v, 2, rz))
