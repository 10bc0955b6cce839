"""The component labelling at each of its tile depths (csrc/ccl.cu: 8, 16 and 32 slices by how many tiles there are) and
the sweeps of csrc/sweep.cu (the Hessian with its slices split among blocks, the DoG in both its tiles), around their ends,
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


@pytest.mark.gpu
@pytest.mark.parametrize("sig", [(2.0, 1.5, 3.2, 2.4), (4.0, 1.8, 6.0, 2.7)])
@pytest.mark.parametrize("W,H,D", [(640, 365, 5), (641, 361, 12), (1283, 192, 11), (639, 383, 23), (67, 47, 13), (70, 25, 1)])
def test_gpu_dog_sweep_tiles(W, H, D, sig):
    """32 x 24 tiles (at least 304 of them) and 32 x 16 ones, rows and columns left over on every side, depths around
    one turn of the z register (11)."""
    import hdog
    norm = np.random.default_rng(W + H + D).normal(0, 1, (D, H, W)).astype(np.float32)
    norm[D // 2, H // 2, W // 2] = np.inf
    norm[0, 1, 2] = np.nan
    p = hdog.make_params(width=W, height=H, depth=D, sigma_xy_small=sig[0], sigma_z_small=sig[1], sigma_xy_large=sig[2],
                         sigma_z_large=sig[3])
    with hdog.Context(p) as ctx:
        got = ctx.dog(torch.from_numpy(norm).cuda()).cpu().numpy()
    ref = orc.dog(norm, *sig)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), ref[~nan].view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(1280, 1712, 4), (1283, 1701, 5)])
def test_gpu_records_over_two_row_threads(W, H, D):
    """Enough 32 x 16 tiles (4256) for the Hessian sweep's two-row form, with an odd last row and a padded width."""
    import hdog
    rng = np.random.default_rng(W + D)
    vol = np.clip(300 + 60 * rng.normal(size=(D, H, W)), 0, 65535).astype(np.uint16)
    p = hdog.make_params(width=W, height=H, depth=D, left_margin=0, right_margin=0, top_margin=0, bottom_margin=0,
                         extra_depth_margin=0, radius_norm_xy=6, radius_norm_z=2, min_intensity=0, min_size=0)
    with hdog.Context(p) as ctx:
        got = ctx.run_substack(torch.from_numpy(vol).cuda(), D, 0)
    ref = orc.substack(orc.params_from(p), vol, D, 0)[0]
    assert len(got) == len(ref)
    for f in ("local_x", "local_y", "local_z", "intensity", "size"):
        assert np.array_equal(got[f], ref[f]), f
