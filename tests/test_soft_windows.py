"""The differentiable chain's window passes (csrc/soft.cu: k_soft_ext_rows / _cols, their adjoints, k_soft_box_x /
_cols, and the *_far kernels) at reaches and line lengths around their blocks (8 entries), groups (reach 31), rings
and tiles, against the FP64 reference.  Every voxel has a fractional part, so no window has a tie.  Bounds as in
test_soft.py (loss 1e-5, input gradients 1e-4 of the largest; sigma gradients 2e-4, its bound for wide windows)."""
import numpy as np
import pytest
import torch

from oracle import soft_ref as sr

SIGMA = [1.2, 1.3, 1.1, 1.9, 2.1, 1.7]
CASES = [
    # D, H, W, rxy, rz
    (9, 20, 33, 0, 2), (9, 20, 33, 1, 0), (12, 30, 41, 3, 3), (11, 17, 66, 4, 4), (16, 40, 29, 5, 1), (20, 36, 47, 7, 6),
    (5, 9, 259, 8, 2), (6, 150, 12, 10, 5), (40, 13, 70, 30, 9), (7, 35, 128, 31, 3), (7, 70, 40, 32, 16), (4, 20, 300, 127, 2),
    (4, 18, 60, 256, 3), (3, 15, 31, 400, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("D,H,W,rxy,rz", CASES)
def test_gpu_windows_match_the_reference(D, H, W, rxy, rz):
    import hdog
    rng = np.random.default_rng(D * 10007 + H * 101 + W + rxy)
    vol = 100 + rng.normal(0, 8, (D, H, W)) + rng.uniform(0, 1, (D, H, W))
    zz, yy, xx = np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij")
    pos = np.stack([rng.integers(0, n, 5) for n in (D, H, W)], 1).astype(np.int32)
    for z, y, x in pos:
        vol += 600 * np.exp(-((xx - x) ** 2 + (yy - y) ** 2) / 9.0 - (zz - z) ** 2 / 5.0)
    vol = vol.astype(np.float32)
    neg = np.stack([rng.integers(0, n, 6) for n in (D, H, W)], 1).astype(np.int32)
    tau = 0.05
    I = torch.tensor(vol, dtype=torch.float64, requires_grad=True)
    sig = torch.tensor(SIGMA, dtype=torch.float32).double().requires_grad_(True)
    L = sr.loss(I, list(sig), torch.tensor(pos, dtype=torch.long), torch.tensor(neg, dtype=torch.long), rxy, rz, 50.0, tau)
    if not torch.isfinite(L):
        pytest.fail("the case has a window without contrast")
    L.backward()
    v = torch.tensor(vol, device="cuda", requires_grad=True)
    s = torch.tensor(SIGMA, dtype=torch.float32, requires_grad=True)
    loss = hdog.soft.soft_loss(v, s, torch.tensor(pos, device="cuda"), torch.tensor(neg, device="cuda"), radius_norm_xy=rxy,
                               radius_norm_z=rz, min_intensity=50.0, tau=tau)
    loss.backward()
    assert abs(float(loss.detach()) - float(L.detach())) <= 1e-5 * max(abs(float(L.detach())), 0.1)
    gs, gI = sig.grad.numpy(), I.grad.numpy()
    assert np.all(np.abs(s.grad.numpy() - gs) <= 2e-4 * np.abs(gs).max()), (s.grad.numpy(), gs)
    assert np.abs(v.grad.cpu().numpy() - gI).max() <= 1e-4 * np.abs(gI).max()
