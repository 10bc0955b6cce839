"""The window adjoints (csrc/soft.cu) where windows hold their extreme several times: each window's gradient goes to its
first one along the axis, x, then y, then z.  The FP64 reference with that rule in its min / max windows; bounds as
in test_soft_windows.py."""
import numpy as np
import pytest
import torch

from oracle import soft_ref as sr

SIGMA = [1.2, 1.3, 1.1, 1.9, 2.1, 1.7]


def first_extreme(x, axis, r, is_max):
    if r == 0:
        return x
    v = x.movedim(axis, -1)
    n = v.shape[-1]
    at = np.clip(np.arange(n)[:, None] + np.arange(-r, r + 1)[None], 0, n - 1)
    win = v.detach().numpy()[..., at]
    k = (win.argmax if is_max else win.argmin)(-1)          # the first of equals
    return v.gather(-1, torch.from_numpy(at[np.arange(n), k])).movedim(-1, axis)


@pytest.mark.gpu
@pytest.mark.parametrize("D,H,W,rxy,rz", [(9, 20, 33, 2, 3), (6, 40, 66, 4, 1), (20, 36, 47, 7, 6), (5, 9, 259, 8, 2),
                                          (40, 13, 70, 30, 9), (7, 70, 40, 32, 16), (4, 20, 300, 127, 2), (2, 300, 20, 31, 1)])
def test_gpu_ties_go_to_the_first_extreme(monkeypatch, D, H, W, rxy, rz):
    import hdog
    monkeypatch.setattr(sr, "minmax1d", first_extreme)
    rng = np.random.default_rng(D * 101 + W)
    vol = rng.integers(100, 112, (D, H, W)).astype(np.float32)
    pos = np.stack([rng.integers(0, n, 9) for n in (D, H, W)], 1).astype(np.int32)
    neg = np.stack([rng.integers(0, n, 7) for n in (D, H, W)], 1).astype(np.int32)
    I = torch.tensor(vol, dtype=torch.float64, requires_grad=True)
    sig = torch.tensor(SIGMA, dtype=torch.float32).double().requires_grad_(True)
    sr.loss(I, list(sig), torch.tensor(pos, dtype=torch.long), torch.tensor(neg, dtype=torch.long), rxy, rz, 50.0,
            0.05).backward()
    v = torch.tensor(vol, device="cuda", requires_grad=True)
    s = torch.tensor(SIGMA, dtype=torch.float32, requires_grad=True)
    hdog.soft.soft_loss(v, s, torch.tensor(pos, device="cuda"), torch.tensor(neg, device="cuda"), radius_norm_xy=rxy,
                        radius_norm_z=rz, min_intensity=50.0, tau=0.05).backward()
    g = I.grad.numpy()
    assert np.isfinite(g).all() and np.abs(g).max() > 0
    assert np.all(np.abs(s.grad.numpy() - sig.grad.numpy()) <= 2e-4 * np.abs(sig.grad.numpy()).max())
    assert np.abs(v.grad.cpu().numpy() - g).max() <= 1e-4 * np.abs(g).max()
