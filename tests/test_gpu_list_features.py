"""The Hessian elements of the foreground list (csrc/sweep.cu) through the records' structureness and blobness: split slices,
one and two rows per thread, padded widths, the separate DoG passes; volumes with nuclei, against the oracle.

The oracle sums the elements in float32, the library in fixed point: with sums off by a share e of the largest
eigenvalue, structureness (the sum of the eigenvalues' squares) is off by about 2 e of itself.  Blobness is l2^2 / (l0 l1) of
negative eigenvalues |l0| >= |l1| >= |l2|, so |l2| is at least blobness |l0| and the error at most 3 sqrt(3) e, absolute.
Regions of some hundred voxels keep e below 1e-5."""
import numpy as np
import pytest
import torch

from helpers import volume
from oracle import oracle as orc

STD, NARROW, WIDE = (2.0, 1.5, 3.2, 2.4), (0.9, 0.8, 1.2, 1.1), (3.0, 1.2, 7.4, 4.3)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,sig", [
    (130, 70, 12, STD), (128, 72, 26, STD), (300, 64, 49, STD), (97, 41, 24, NARROW), (101, 75, 30, WIDE),   # split slices
    (640, 365, 8, STD), (641, 361, 13, STD),                                                        # one row
    (1280, 1712, 6, STD), (1283, 1701, 7, STD)])                                                    # two rows
def test_gpu_structureness_and_blobness(W, H, D, sig):
    import hdog
    vol = volume(W, H, D)
    p = hdog.make_params(width=W, height=H, depth=D, left_margin=0, right_margin=0, top_margin=0, bottom_margin=0,
                         extra_depth_margin=-int(2 * sig[3] + 0.5), radius_norm_xy=20, radius_norm_z=3, min_intensity=50, min_size=4,
                         sigma_xy_small=sig[0], sigma_z_small=sig[1], sigma_xy_large=sig[2], sigma_z_large=sig[3])
    with hdog.Context(p) as ctx:
        got = ctx.run_substack(torch.from_numpy(vol).cuda(), D, 0)
    ref = orc.substack(orc.params_from(p), vol, D, 0)[0]
    assert len(ref) > 5
    assert len(got) == len(ref)
    for f in ("local_x", "local_y", "local_z", "intensity", "size"):
        assert np.array_equal(got[f].view(np.uint32) if f == "intensity" else got[f],
                              ref[f].view(np.uint32) if f == "intensity" else ref[f]), f
    st, bl = ([r[f].astype(np.float64) for r in (got, ref)] for f in ("structureness", "blobness"))
    assert np.all(np.abs(st[0] - st[1]) <= 1e-4 * st[1])
    assert np.all(np.abs(bl[0] - bl[1]) <= 1e-4)
