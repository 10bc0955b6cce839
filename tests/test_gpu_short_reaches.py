"""The normalization's and the erosion's y and x passes at reaches below 4 (csrc/norm.cu: k_mm_y_short, k_erode_x_quad and, on other widths, k_mm_x),
bit for bit against the oracle: lines shorter than a window, and around a warp's 32 columns and a block's 64 rows."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

SHAPES = [(2, 2, 1), (5, 3, 2), (31, 63, 4), (33, 65, 3), (64, 130, 5), (259, 8, 7)]


def volume(W, H, D):
    rng = np.random.default_rng(W * 7919 + H * 31 + D)
    return (rng.integers(0, 65536, (D, H, W)) // rng.integers(1, 200, (D, H, W))).astype(np.uint16)


@pytest.mark.gpu
@pytest.mark.parametrize("rxy", [0, 1, 2, 3])
@pytest.mark.parametrize("W,H,D", SHAPES)
def test_gpu_erosion_matches_the_oracle(W, H, D, rxy):
    import hdog
    vol = volume(W, H, D)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        got = ctx.erosion(torch.from_numpy(vol).cuda(), rxy, 1).cpu().numpy()
    assert np.array_equal(got, orc.erosion(vol, rxy, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("rxy", [1, 2, 3])
@pytest.mark.parametrize("W,H,D", SHAPES)
def test_gpu_normalize_matches_the_oracle(W, H, D, rxy):
    import hdog
    vol = volume(W, H, D)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=rxy, radius_norm_z=2, min_intensity=20)) as ctx:
        got = ctx.normalize(torch.from_numpy(vol).cuda()).cpu().numpy()
    ref = orc.normalize(vol, rxy, 2, 20.0)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
