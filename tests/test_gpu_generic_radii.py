"""The DoG passes at known and at other reaches (csrc/dog.cu), and the chain on frames of any width: rows of the
normalized and the DoG volume are padded to 4 there, the mask's are not.  DoG volumes bit for bit and records
against the oracle, at radii around the instantiations (1, 2, 14, 15; the small scale the wider one), widths of
every remainder, and through the dense region pass (the stage call)."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

SIGMAS = [(0.4, 0.4, 0.6, 0.7), (0.9, 0.8, 1.2, 1.1), (2.9, 1.9, 7.1, 3.1), (3.0, 1.2, 7.4, 4.3), (3.2, 2.4, 2.0, 1.5)]


def volume(W, H, D):
    rng = np.random.default_rng(W * 1009 + H * 17 + D)
    v = 100 + rng.normal(0, 8, (D, H, W))
    zz, yy, xx = np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij")
    for _ in range(max(3, W * H * D // 6000)):
        z, y, x = rng.integers(0, D), rng.integers(0, H), rng.integers(0, W)
        v += rng.uniform(200, 2000) * np.exp(-((xx - x) ** 2 + (yy - y) ** 2) / 12.0 - (zz - z) ** 2 / 5.0)
    return np.clip(np.rint(v), 0, 65535).astype(np.uint16)


def make(hdog, W, H, D, sig, **kw):
    return hdog.make_params(width=W, height=H, depth=D, left_margin=0, right_margin=0, top_margin=0, bottom_margin=0,
                            extra_depth_margin=0, radius_norm_xy=6, radius_norm_z=2, min_intensity=50, min_size=0,
                            sigma_xy_small=sig[0], sigma_z_small=sig[1], sigma_xy_large=sig[2], sigma_z_large=sig[3], **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("sig", SIGMAS)
@pytest.mark.parametrize("W,H,D", [(131, 34, 9), (64, 33, 21), (258, 9, 12), (5, 40, 8)])
def test_gpu_dog_matches_the_oracle(sig, W, H, D):
    import hdog
    norm = np.random.default_rng(W + D).normal(0, 1, (D, H, W)).astype(np.float32)
    norm[D // 2, H // 2, W // 2] = np.inf
    norm[0, 1, 2] = np.nan
    with hdog.Context(make(hdog, W, H, D, sig)) as ctx:
        got = ctx.dog(torch.from_numpy(norm).cuda()).cpu().numpy()
    ref = orc.dog(norm, *sig)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), ref[~nan].view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("sig", [SIGMAS[1], SIGMAS[3], (2.0, 1.5, 3.2, 2.4)])
@pytest.mark.parametrize("W,H,D", [(97, 41, 24), (98, 37, 20), (99, 40, 22), (100, 39, 24), (34, 30, 20)])
def test_gpu_records_match_the_oracle(sig, W, H, D):
    import hdog
    vol = volume(W, H, D)
    p = make(hdog, W, H, D, sig)
    with hdog.Context(p) as ctx:
        dv = torch.from_numpy(vol).cuda()
        got = ctx.run_substack(dv, D, 0)
        norm = ctx.normalize(dv)
        dog = ctx.dog(norm)
        mask, _ = ctx.hessian_pd(dog)
        labels = ctx.ccl(mask)
        reg = ctx.regional_features(labels, norm, dog)
    ref = orc.substack(orc.params_from(p), vol, D, 0)[0]
    assert len(got) == len(ref)
    for f in ("local_x", "local_y", "local_z", "intensity", "size"):
        assert np.array_equal(got[f], ref[f]), f
    R = orc.regions(labels.cpu().numpy(), norm.cpu().numpy(), dog.cpu().numpy())
    assert reg["num_regions"] == R["num_regions"]
    assert np.array_equal(reg["count"][1:], R["count"][1:].astype(np.uint32))
    assert np.array_equal(reg["intensity"][1:].view(np.uint32), R["max_norm"][1:].view(np.uint32))
    scale = np.abs(R["hess_f64"][:, 1:]).max(axis=0) if R["num_regions"] > 1 else np.zeros(0)
    for k in range(6):
        assert np.all(np.abs(reg["hessian"][k, 1:].astype(np.float64) - R["hess_f64"][k, 1:]) <= 1e-6 * scale + 1e-30)
