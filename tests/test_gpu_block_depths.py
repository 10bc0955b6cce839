"""The component labelling at each of its tile depths (csrc/ccl.cu: 8, 16 and 32 slices by how many tiles there are) and
the Hessian sweep with its slices split among blocks (csrc/sweep.cu), at depths around a tile's and a piece's end,
against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("density", [0.04, 0.3, 1.0])
@pytest.mark.parametrize("W,H,D", [(70, 20, 7), (64, 16, 8), (65, 17, 9), (130, 50, 33),          # 8 slices
                                   (640, 128, 16), (641, 127, 17), (600, 130, 35),                 # 16 slices
                                   (640, 256, 33), (1283, 321, 31)])                               # 32 slices
def test_gpu_labels_match_the_oracle(W, H, D, density):
    import hdog
    rng = np.random.default_rng(W + 3 * H + 7 * D)
    mask = (rng.random((D, H, W)) < density).astype(np.uint8)
    if density == 1.0:   # one spiral through every slice and walls across every tile
        mask[:, ::2, 1:] = 0
        mask[1::2, :, : W // 2] = 0
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        got = ctx.ccl(torch.from_numpy(mask).cuda()).cpu().numpy()
    assert np.array_equal(got, orc.ccl(mask)[0])


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(64, 16, 5), (67, 18, 11), (130, 35, 12), (128, 34, 13), (61, 33, 25), (300, 64, 49)])
def test_gpu_records_over_split_slices(W, H, D):
    import hdog
    rng = np.random.default_rng(W + H + D)
    vol = np.clip(300 + 60 * rng.normal(size=(D, H, W)), 0, 65535).astype(np.uint16)
    p = hdog.make_params(width=W, height=H, depth=D, left_margin=0, right_margin=0, top_margin=0, bottom_margin=0,
                         extra_depth_margin=0, radius_norm_xy=6, radius_norm_z=2, min_intensity=0, min_size=0)
    with hdog.Context(p) as ctx:
        got = ctx.run_substack(torch.from_numpy(vol).cuda(), D, 0)
    ref = orc.substack(orc.params_from(p), vol, D, 0)[0]
    assert len(got) == len(ref)
    for f in ("local_x", "local_y", "local_z", "intensity", "size"):
        assert np.array_equal(got[f], ref[f]), f
