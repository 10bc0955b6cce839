"""The differentiable chain at few and at many sample points (csrc/soft.cu: points_local): with few, the
DoG is evaluated at the points' own neighbourhoods, with many over the whole volume.

Repeating every point leaves the loss and its gradients as they are (they are means), and
enough repeats take the call from the first form to the second, so both are held to the FP64
reference and, through it, to each other.  Points lie in the corners, on the faces and inside;
radii differ per axis and scale.  Bounds as in test_soft.py (loss 1e-5, threshold gradients and input
gradients 1e-4, sigma gradients 2e-4 relative, the bound for wide windows there).
"""
import ctypes

import numpy as np
import pytest
import torch

from oracle import soft_ref as sr

CASES = [
    # D, H, W, sigmas, (rxy, rz)
    (14, 40, 44, [1.2, 1.3, 1.1, 1.9, 2.1, 1.7], (4, 2)),
    (9, 21, 35, [0.6, 2.2, 0.9, 3.4, 1.1, 1.4], (5, 1)),
    (24, 33, 29, [2.0, 1.6, 2.4, 2.6, 3.3, 0.7], (3, 3)),
]
TAU = 0.05


def make(D, H, W):
    rng = np.random.default_rng(D * 1000 + W)
    vol = 100 + rng.normal(0, 8, (D, H, W)) + rng.uniform(0, 1, (D, H, W))
    zz, yy, xx = np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij")
    centres = [(0, 0, 0), (D - 1, H - 1, W - 1), (D // 2, H // 2, W // 2), (D // 3, H - 4, 3), (D - 2, 2, W // 2)]
    for c in centres:
        vol += 500 * np.exp(-((xx - c[2]) ** 2 + (yy - c[1]) ** 2) / 9.0 - (zz - c[0]) ** 2 / 5.0)
    pos = np.array(centres + [(0, H // 2, W - 1), (1, 1, 1)], np.int32)
    neg = np.stack([rng.integers(0, n, 6) for n in (D, H, W)], 1).astype(np.int32)
    return vol.astype(np.float32), pos, neg


def reference(vol, pos, neg, sigma, r, b):
    I = torch.tensor(vol, dtype=torch.float64, requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float32).double().requires_grad_(True)
    bt = torch.tensor(b, dtype=torch.float32).double().requires_grad_(True)
    L = sr.loss(I, list(s), torch.tensor(pos, dtype=torch.long), torch.tensor(neg, dtype=torch.long), r[0], r[1], 50.0,
                TAU, b=list(bt))
    L.backward()
    return float(L.detach()), I.grad.numpy(), s.grad.numpy(), bt.grad.numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("repeat,keep", [(1, True), (1, False), (4000, True), (4000, False)])
def test_gpu_points_local_and_dense_match_the_reference(case, repeat, keep):
    import hdog
    D, H, W, sigma, r = CASES[case]
    vol, pos, neg = make(D, H, W)
    b = [0.01, -0.0005, 0.00002]
    L, gI, gs, gb = reference(vol, pos, neg, sigma, r, b)
    v = torch.tensor(vol, device="cuda", requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float32, requires_grad=True)
    bt = torch.tensor(b, dtype=torch.float32, requires_grad=True)
    p, n = (torch.tensor(np.tile(a, (repeat, 1)), device="cuda") for a in (pos, neg))
    loss = hdog.soft.soft_loss(v, s, p, n, thresh=bt, radius_norm_xy=r[0], radius_norm_z=r[1], min_intensity=50.0,
                               tau=TAU, keep_intermediates=keep)
    loss.backward()
    assert abs(float(loss.detach()) - L) <= 1e-5 * abs(L), (float(loss.detach()), L)
    assert np.all(np.abs(s.grad.numpy() - gs) <= 2e-4 * np.abs(gs).max()), (s.grad.numpy(), gs)
    assert np.all(np.abs(bt.grad.numpy() - gb) <= 1e-4 * np.abs(gb).max()), (bt.grad.numpy(), gb)
    assert np.abs(v.grad.cpu().numpy() - gI).max() <= 1e-4 * np.abs(gI).max()


@pytest.mark.gpu
def test_gpu_kept_workspace_of_a_call_with_few_points_serves_one_with_many():
    import hdog
    from hdog.soft import _params
    D, H, W, sigma, r = CASES[0]
    vol, pos, neg = make(D, H, W)
    v = torch.tensor(vol, device="cuda")
    prm = _params(v, torch.tensor(sigma), torch.zeros(3), (r[0], r[1], 50.0, TAU, 1.0))
    L = hdog.lib()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def grads(first, then):
        ws = torch.empty(L.hdog_soft_workspace_bytes(ctypes.byref(prm)), dtype=torch.uint8, device="cuda")
        loss, gv = torch.empty(1, device="cuda"), torch.empty_like(v)
        gs, gb = torch.empty(6, device="cuda"), torch.empty(3, device="cuda")
        p, n = (torch.tensor(np.tile(a, (first, 1)), device="cuda") for a in (pos, neg))
        q = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        hdog.check(L.hdog_soft_forward(ctypes.byref(prm), q(v), q(p), len(p), q(n), len(n), q(loss), None, q(ws), st))
        p2, n2 = (torch.tensor(np.tile(a, (then, 1)), device="cuda") for a in (pos, neg))
        hdog.check(L.hdog_soft_backward_kept(ctypes.byref(prm), q(v), q(p2), len(p2), q(n2), len(n2), 1.0, q(gv), q(gs),
                                             q(gb), q(ws), st))
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in (gv, gs, gb)]

    base = grads(1, 1)
    for first, then in ((1, 4000), (4000, 1), (4000, 4000)):
        for a, x in zip(base, grads(first, then)):
            assert np.abs(a - x).max() <= 2e-4 * np.abs(a).max(), (first, then)
