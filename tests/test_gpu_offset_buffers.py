"""Stage calls on buffers that start inside an allocation: a mask on any byte, labels, volumes on any of their elements.
Widths whose rows the labelling reads two and sixteen voxels at a time and writes four at a time; against the oracle and
the same calls on aligned buffers."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc


def at(a, off, fill=0):
    """The array's values on the device, `off` elements into an allocation."""
    t = torch.from_numpy(a)
    buf = torch.full((a.size + off + 8,), fill, dtype=t.dtype, device="cuda")
    v = buf[off:off + a.size].view(a.shape)
    v.copy_(t)
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(114, 86, 2), (64, 33, 9), (192, 20, 17), (67, 31, 5)])
@pytest.mark.parametrize("off", [1, 2, 3, 4, 8])
def test_gpu_labels_of_offset_buffers(W, H, D, off):
    import hdog
    mask = (np.random.default_rng(W + off).random((D, H, W)) < 0.3).astype(np.uint8)
    want = orc.ccl(mask)[0]
    with hdog.Context(hdog.make_params(width=W, height=H, depth=D)) as ctx:
        m = at(mask, off)
        out = at(np.full((D, H, W), -7, np.int32), off % 4, -7)
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        q = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        hdog.check(hdog.lib().hdog_ccl(ctx._h, q(m), q(out), st))
        assert np.array_equal(out.cpu().numpy(), want)
        out.fill_(-7)
        hdog.check(hdog.lib().hdog_ccl_noalloc(q(m), q(out), W, H, D, st))
        assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D", [(114, 46, 6), (64, 33, 9), (67, 31, 5)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_gpu_stages_of_offset_buffers(W, H, D, off):
    import hdog
    rng = np.random.default_rng(W + off)
    img = rng.integers(0, 5000, (D, H, W)).astype(np.uint16)
    f = rng.normal(0, 1, (D, H, W)).astype(np.float32)
    lab = orc.ccl((rng.random((D, H, W)) < 0.3).astype(np.uint8))[0]
    p = hdog.make_params(width=W, height=H, depth=D, radius_norm_xy=6, radius_norm_z=2, min_intensity=50, sigma_xy_small=2.0,
                         sigma_z_small=1.5, sigma_xy_large=3.2, sigma_z_large=2.4)
    with hdog.Context(p) as ctx:
        def run(o):
            norm, dog, g = at(f, o), at(f, o), at(f[::-1].copy(), o)
            reg = ctx.regional_features(at(lab, o), g, dog)
            return [ctx.normalize(at(img, o)).cpu().numpy(), ctx.erosion(at(img, o), 2, 1).cpu().numpy(),
                    ctx.erosion(at(img, o), 9, 1).cpu().numpy(), ctx.dog(norm).cpu().numpy(),
                    ctx.hessian_pd(dog, want_hessian=True)[1].cpu().numpy()] + [np.asarray(reg[k]) for k in sorted(reg)]
        for a, b in zip(run(0), run(off)):
            assert a.tobytes() == b.tobytes()
