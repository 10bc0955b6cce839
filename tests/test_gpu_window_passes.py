"""The normalization's and the erosion's window passes (csrc/norm.cu: k_mm_z_stream, k_mm_y_cols, k_mm_x_rows)
bit for bit against the oracle, at reaches around their block and ring sizes (8 and 16 entries, 127 and 255) and at
lines shorter and longer than a window and than the row pass's chunks of 256."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

CASES = [
    # W, H, D, rxy, rz
    (67, 45, 13, 4, 1), (256, 33, 7, 7, 2), (257, 64, 5, 8, 3), (31, 129, 9, 9, 4), (300, 257, 4, 15, 5), (129, 40, 20, 16, 6),
    (64, 300, 18, 20, 7), (515, 21, 17, 31, 8), (90, 131, 3, 33, 9), (700, 50, 2, 100, 5), (20, 400, 2, 127, 1), (513, 30, 3, 128, 3),
    (5, 3, 2, 12, 4), (2, 2, 1, 5, 1),
]


def volume(W, H, D):
    rng = np.random.default_rng(W * 7919 + H * 31 + D)
    v = rng.integers(0, 65536, (D, H, W)) // rng.integers(1, 200, (D, H, W))
    return v.astype(np.uint16)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,rxy,rz", CASES)
def test_gpu_normalize_matches_the_oracle(W, H, D, rxy, rz):
    import hdog
    vol = volume(W, H, D)
    p = hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=rxy, radius_norm_z=rz, min_intensity=20)
    with hdog.Context(p) as ctx:
        got = ctx.normalize(torch.from_numpy(vol).cuda()).cpu().numpy()
    ref = orc.normalize(vol, rxy, rz, 20.0)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,rxy,rz", CASES + [(600, 20, 2, 255, 2), (300, 520, 1, 256, 0)])
def test_gpu_erosion_matches_the_oracle(W, H, D, rxy, rz):
    import hdog
    vol = volume(W, H, D)
    p = hdog.make_params(width=W, height=H, depth=D)
    with hdog.Context(p) as ctx:
        got = ctx.erosion(torch.from_numpy(vol).cuda(), rxy, rz).cpu().numpy()
    assert np.array_equal(got, orc.erosion(vol, rxy, rz))
