"""The region sums without a list (csrc/regions.cu, k_accumulate): one region in every voxel, runs of a few voxels and of
one, components, on frames of 2^16 and more along each axis (the packed coordinate sums), against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc


def labels_of(kind, W, H, D, rng):
    n = W * H * D
    if kind == "components":
        return orc.ccl((rng.random((D, H, W)) < 0.2).astype(np.uint8))[0]
    if kind == "one":
        lab = np.ones(n, np.int32)
    else:   # random labels in runs of 1 or 5 voxels; voxels 1 .. 39 are their regions' roots
        run = 5 if kind == "runs" else 1
        lab = np.repeat(rng.integers(1, 40, n // run + 1), run)[:n].astype(np.int32)
        lab[:40] = np.arange(40)
    lab[0] = 0
    return lab.reshape(D, H, W)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["components", "one", "runs", "mixed"])
@pytest.mark.parametrize("W,H,D", [(70003, 6, 3), (6, 70003, 3), (5, 7, 70003), (641, 40, 9), (30, 5, 3)])
def test_gpu_region_sums(W, H, D, kind):
    import hdog
    rng = np.random.default_rng(W + H)
    lab = labels_of(kind, W, H, D, rng)
    norm = rng.normal(0, 1, (D, H, W)).astype(np.float32)
    dog = rng.normal(0, 1e-2, (D, H, W)).astype(np.float32)
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        G = ctx.regional_features(*(torch.from_numpy(a).cuda() for a in (lab, norm, dog)))
    R = orc.regions(lab, norm, dog)
    assert G["num_regions"] == R["num_regions"]
    assert np.array_equal(G["label"][1:], R["label"][1:])
    assert np.array_equal(G["count"][1:], R["count"][1:].astype(np.uint32))
    assert np.array_equal(G["intensity"][1:].view(np.uint32), R["max_norm"][1:].view(np.uint32))
    c16 = (R["count"][1:] & 0xFFFF).astype(np.float32)
    with np.errstate(divide="ignore", invalid="ignore"):
        for k in range(3):
            cent = (R["sum_xyz"][k, 1:].astype(np.float32) / c16).astype(np.float32)
            assert np.array_equal(G["centroid"][k, 1:].view(np.uint32), cent.view(np.uint32)), k
    # fixed point with 36 fractional bits: half a unit a voxel, and one float rounding
    bound = R["count"][1:] * 2.0 ** -37
    for k in range(6):
        d = np.abs(G["hessian"][k, 1:].astype(np.float64) - R["hess_f64"][k, 1:])
        assert np.all(d <= bound + 2.0 ** -23 * np.abs(R["hess_f64"][k, 1:])), k
