"""The row passes (csrc/window.cuh) at both their lane counts and beside the tiles that very long rows take: frames
around the rules' lines, at reaches from both sides of each, bit for bit against the oracle; the differentiable
chain's extremes through its loss and gradients against the FP64 reference."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from oracle import soft_ref as sr

# width, height, depth: 32 lanes (few rows), tiles (long rows), 8 lanes (many rows; wide and narrow)
FRAMES = [(300, 40, 3), (129, 61, 2), (2600, 9, 2), (6000, 5, 2), (20011, 3, 3), (70, 250, 20), (131, 304, 16), (1030, 608, 16)]


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", FRAMES)
@pytest.mark.parametrize("r", [4, 5, 6, 7, 16, 31, 32])
def test_gpu_rows_match_the_oracle(W, H, D, r):
    import hdog
    if W * H * D > 2e6 and r not in (6, 31):
        pytest.skip("large frame: two reaches")
    rng = np.random.default_rng(W + r)
    v = rng.integers(0, 65536, (D, H, W)).astype(np.uint16)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=r, radius_norm_z=1, min_intensity=50,
                                       sigma_z_small=0.1, sigma_z_large=0.2, extra_depth_margin=0)) as ctx:
        d = torch.from_numpy(v).cuda()
        norm = ctx.normalize(d).cpu().numpy()
        ero = ctx.erosion(d, r, 1).cpu().numpy()
    assert np.array_equal(norm.view(np.uint32), orc.normalize(v, r, 1, 50.0).view(np.uint32))
    assert np.array_equal(ero, orc.erosion(v, r, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("D,H,W,r", [(2, 30, 200, 6), (2, 5, 3000, 9), (20, 250, 40, 6), (3, 20, 150, 31)])
def test_gpu_soft_rows_match_the_reference(D, H, W, r):
    import hdog
    rng = np.random.default_rng(D + W)
    vol = (100 + rng.uniform(0, 900, (D, H, W))).astype(np.float32)
    pos = np.stack([rng.integers(0, n, 9) for n in (D, H, W)], 1).astype(np.int32)
    neg = np.stack([rng.integers(0, n, 7) for n in (D, H, W)], 1).astype(np.int32)
    sigma = [1.0, 1.0, 0.8, 1.6, 1.6, 1.3]
    I = torch.tensor(vol, dtype=torch.float64, requires_grad=True)
    s64 = torch.tensor(sigma, dtype=torch.float32).double().requires_grad_(True)
    L = sr.loss(I, list(s64), torch.tensor(pos, dtype=torch.long), torch.tensor(neg, dtype=torch.long), r, 1, 50.0, 0.05)
    L.backward()
    v = torch.tensor(vol, device="cuda", requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float32, requires_grad=True)
    loss = hdog.soft.soft_loss(v, s, torch.tensor(pos, device="cuda"), torch.tensor(neg, device="cuda"), radius_norm_xy=r,
                               radius_norm_z=1, min_intensity=50.0, tau=0.05)
    loss.backward()
    # the chain's bounds (test_soft_points.py), the loss against the scores' scale of 1 / 8
    assert abs(float(loss.detach()) - float(L.detach())) <= 1e-5 * 0.125
    assert np.all(np.abs(s.grad.numpy() - s64.grad.numpy()) <= 2e-4 * np.abs(s64.grad.numpy()).max())
    gI = I.grad.numpy()
    assert np.abs(v.grad.cpu().numpy() - gI).max() <= 1e-4 * np.abs(gI).max()
