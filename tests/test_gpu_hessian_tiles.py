"""The Hessian stage (csrc/dog.cu, k_hessian_pd) with blocks of 8 and 16 slices, quads and single columns staged, frames
that end inside a tile on every side: mask and the six planes bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(33, 31, 29), (101, 75, 5), (32, 8, 8), (36, 9, 9), (5, 6, 17), (2, 2, 1),       # 8 slices
                                   (640, 250, 17), (641, 251, 16), (399, 403, 33)])                              # 16
def test_gpu_hessian_stage(W, H, D):
    import hdog
    dog = np.random.default_rng(W + H + D).normal(0, 1e-2, (D, H, W)).astype(np.float32)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        mask, hess = ctx.hessian_pd(torch.from_numpy(dog).cuda(), want_hessian=True)
    ref, h6 = orc.hessian_pd(dog, want_hessian=True)
    assert np.array_equal(mask.cpu().numpy(), ref)
    assert np.array_equal(hess.cpu().numpy().view(np.uint32), h6.view(np.uint32))
