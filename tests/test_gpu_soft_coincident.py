"""Many points at one place, in volumes large enough that the DoG is still evaluated at the points (csrc/soft.cu,
points_local): the loss is a mean, so its gradients are those of a single point there.  Only roundings of 1 / n and of single
terms differ, a few parts in 10^7; the bound is the chain's 1e-4 halved twice."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("keep", [True, False])
def test_gpu_coincident_points_in_a_large_volume(keep):
    import hdog
    D, H, W = 48, 400, 512
    gen = torch.Generator(device="cuda").manual_seed(3)
    vol = torch.rand((D, H, W), generator=gen, device="cuda") * 900 + 100
    pos = torch.tensor([[D // 2, 201, 301]], dtype=torch.int32, device="cuda")
    neg = torch.tensor([[D // 2 + 1, 60, 70]], dtype=torch.int32, device="cuda")

    def grads(n):
        v = vol.clone().requires_grad_(True)
        s = torch.tensor([1.0] * 3 + [1.6] * 3, requires_grad=True)
        b = torch.zeros(3, requires_grad=True)
        hdog.soft.soft_loss(v, s, pos.repeat(n, 1), neg, thresh=b, radius_norm_xy=20, radius_norm_z=5, min_intensity=50.0,
                            tau=0.05, keep_intermediates=keep).backward()
        return [t.grad.double().cpu().numpy() for t in (v, s, b)]

    for one, many in zip(grads(1), grads(40000)):
        assert np.abs(one).max() > 0
        assert np.abs(one - many).max() <= 2.5e-5 * np.abs(one).max()
