"""Batches of substacks of a few voxels: the foreground list's roots, one word an entry, lie in a volume that is
smaller than them there."""
import ctypes

import numpy as np
import pytest

import hdog
from oracle import oracle as orc

# width, height, depth
FRAMES = [(2, 2, 4), (5, 4, 5), (4, 4, 6), (7, 6, 5), (8, 8, 8), (9, 8, 8)]


def make(W, H, D):
    return hdog.make_params(width=W, height=H, depth=D, left_margin=0, right_margin=0, top_margin=0, bottom_margin=0,
                            extra_depth_margin=0, radius_norm_xy=2, radius_norm_z=1, min_intensity=0, min_size=0,
                            sigma_xy_small=0.6, sigma_z_small=0.4, sigma_xy_large=1.0, sigma_z_large=0.6)


@pytest.mark.parametrize("W,H,D", FRAMES + [(64, 48, 16), (101, 75, 32)])
@pytest.mark.parametrize("subs", [1, 3, 40])
def test_the_scratch_holds_the_list_its_roots_and_the_edges(W, H, D, subs):
    n = ctypes.c_size_t()
    hdog.check(hdog.lib().hdog_ctx_bytes(ctypes.byref(make(W, H, D)), subs, ctypes.byref(n)))
    voxels = W * H * D
    entries = voxels // 8 + 1024          # of the list (32 bytes), as many roots (4) and at least as many edges (8)
    # the list's counters lie 4096 bytes apart; a voxel takes 2 bytes of input, 8 + 4 + 4 of intermediate volumes, 1 of
    # mask and 4 of labels
    assert n.value >= subs * (entries * (32 + 4 + 8) + 4096 + 23 * voxels)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", FRAMES)
def test_gpu_batches_of_small_frames(W, H, D):
    import torch
    rng = np.random.default_rng(W * 100 + H * 10 + D)
    vol = rng.integers(100, 4000, (70, H, W)).astype(np.uint16)
    p = make(W, H, D)
    want = orc.stack(orc.params_from(p), vol)
    assert len(want) > 0
    for subs in (1, 40):
        with hdog.Context(p, max_substacks=subs) as ctx:
            got = ctx.run_stack(torch.from_numpy(vol).cuda())
        assert len(got) == len(want)
        for f in ("local_x", "local_y", "local_z", "intensity", "size"):
            assert np.array_equal(got[f], want[f]), (subs, f)
