"""The list of cross-tile edges of the labelling (csrc/ccl.cu) with tiles of 8 and 16 slices: dense masks whose edges
32-slice tiles would fit into N/8 stay on the list, denser ones overflow it and are merged from the mask, with the oracle's
labels either way."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,density,overflows", [
    (128, 96, 16, 0.58, False), (131, 77, 33, 0.44, False), (66, 50, 20, 0.47, False), (100, 100, 32, 0.53, False),
    (128, 96, 16, 0.9, True), (131, 77, 33, 0.8, True), (66, 50, 20, 0.6, True), (256, 256, 32, 0.95, True)])
def test_gpu_labels_of_dense_masks(W, H, D, density, overflows):
    import hdog
    mask = (np.random.default_rng(W + D).random((D, H, W)) < density).astype(np.uint8)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        got = ctx.ccl(torch.from_numpy(mask).cuda()).cpu().numpy()
        edges, cap = ctx.ccl_edge_count()
    assert (edges > cap) == overflows, (edges, cap)
    assert np.array_equal(got, orc.ccl(mask)[0])
