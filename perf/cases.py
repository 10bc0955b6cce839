"""The calls whose speed is measured: HDoG detection of whole stacks and single substacks, the
batched graph form, the stage entry points, the differentiable chain and the per-record steps,
each through the package's public interface, from the smallest calls to a full camera stack.

listed() names the measured cases, draw() gives more of the same ranges, prepare() makes a case's
inputs and the contexts that a program keeps, run() is one pass, work() what a pass cannot do
without, exact() the same outputs in 64 bits where they have such values.

Volumes are synthetic light-sheet data with the statistics of hdog.synth (noisy background,
Gaussian nuclei, some in touching pairs, attenuation along z, row striping), made on the GPU from
the seed; nuclei are summed as integers, so the same seed gives the same volume.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cubic-informatics_gb300"))
import hdog  # noqa: E402

# The benchmark's detection parameters and the parameter file's example values.
TUNED = dict(rxy=20, rz=5, sxy1=2.0, sz1=1.5, sxy2=3.2, sz2=2.4, min_intensity=50, margin=100, extra=3, min_size=0)
EXAMPLE = dict(rxy=100, rz=5, sxy1=4.0, sz1=1.8, sxy2=6.0, sz2=2.7, min_intensity=1000, margin=100, extra=3,
               min_size=10)
# Nuclei and background that go with them (hdog.synth's; wider and brighter for the example).
NUCLEI = dict(bg=100.0, bg_sd=8.0, nxy_lo=2.0, nxy_hi=3.5, nz_lo=1.2, nz_hi=2.0, peak_lo=300.0, peak_hi=3000.0)
WIDE_NUCLEI = dict(bg=700.0, bg_sd=40.0, nxy_lo=3.5, nxy_hi=6.0, nz_lo=1.5, nz_hi=2.4, peak_lo=1000.0, peak_hi=8000.0)
SOFT_SIGMA = dict(sx1=2.0, sy1=2.0, sz1=1.5, sx2=3.2, sy2=3.2, sz2=2.4)
SMALL_DENSITY = 400.0 / (256 * 256 * 64)


def _stack(W, H, L, depth, batch, par, nuc, density, host=False, ave=False):
    return dict(kind="stack", W=W, H=H, L=L, depth=depth, batch=batch, density=density, host=host, ave=ave, **par, **nuc)


def listed():
    small = dict(TUNED, margin=10)
    return [
        # one substack of a cropped preview, host memory in and records out: the smallest call, all latency
        dict(_stack(128, 96, 16, 16, 1, dict(small, extra=1, margin=0), NUCLEI, 2e-4, host=True), name="substack_128x96x16"),
        # the 256x256x64 cube that parameters are tried out on, from host memory
        dict(_stack(256, 256, 64, 32, 4, small, NUCLEI, SMALL_DENSITY, host=True), name="cube_256x256x64"),
        # an odd-sized tile with other radii and sigmas, summed intensity (is_ave_mode), already on the GPU
        dict(_stack(683, 517, 75, 32, 4, dict(small, rxy=12, rz=3, sxy1=1.5, sz1=1.2, sxy2=2.4, sz2=1.9), NUCLEI, 6e-5,
                    ave=True), name="stack_683x517x75"),
        # full frames with the example parameter file's radii and sigmas (normalization reach 100)
        dict(_stack(2560, 2160, 64, 32, 4, EXAMPLE, WIDE_NUCLEI, 2e-5), name="example_2560x2160x64"),
        # one camera stack with the benchmark's parameters, on the GPU: the largest call
        dict(_stack(2560, 2160, 128, 32, 8, TUNED, NUCLEI, 60000 / (2560 * 2160 * 128)), name="camera_2560x2160x128"),
        # a half-width stack streamed from page-locked host memory, as a pipeline over a brain feeds it
        dict(_stack(1280, 2160, 160, 32, 8, TUNED, NUCLEI, 6e-5, host=True), name="host_1280x2160x160"),
        # many small stacks of uneven depth and frame through one captured graph
        dict(kind="graph", W=256, H=256, n=12, depth=32, batch=16, density=SMALL_DENSITY, name="graph_12_small", **small, **NUCLEI),
        # the stage entry points one after the other, as the stage-dump programs call them
        dict(kind="stages", W=640, H=720, L=32, density=6e-5, erosion=2, name="stages_640x720x32", **dict(small, rxy=25, rz=4, sxy1=2.5, sz1=1.6,
                                                                                    sxy2=4.0, sz2=2.4), **NUCLEI),
        # forward and backward of the differentiable chain: a crop, where launches count
        dict(kind="soft", W=80, H=72, L=24, rxy=20, rz=5, points=64, keep=True, density=1e-4, name="soft_80x72x24", **SOFT_SIGMA, **NUCLEI),
        # an odd volume, other reaches and sigmas, the forward recomputed in the backward
        dict(kind="soft", W=187, H=203, L=61, rxy=9, rz=3, points=700, keep=False, density=1e-4, name="soft_187x203x61", sx1=1.7, sy1=1.9,
             sz1=1.2, sx2=2.9, sy2=3.0, sz2=2.1, **NUCLEI),
        # the fitting workload: 128x512x512 with 2000 positive and 2000 negative points
        dict(kind="soft", W=512, H=512, L=128, rxy=20, rz=5, points=2000, keep=True, density=3200 / 2 ** 25, name="soft_512x512x128",
             **SOFT_SIGMA, **NUCLEI),
        # the per-record steps after detection, for the records of a large stack
        dict(kind="post", n=400000, ave=False, name="records_400000"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_par(rng):
    sxy1, sz1 = round(rng.uniform(1.2, 4.0), 2), round(rng.uniform(0.9, 2.0), 2)
    ratio = rng.uniform(1.4, 1.7)
    return dict(rxy=_log_int(rng, 5, 100), rz=rng.randint(1, 7), sxy1=sxy1, sz1=sz1, sxy2=round(sxy1 * ratio, 2),
                sz2=round(sz1 * ratio, 2), min_intensity=50, margin=rng.choice([0, 10, 40]), extra=rng.randint(0, 3),
                min_size=rng.choice([0, 10]))


def draw(rng):
    kind = rng.choice(["stack", "stack", "stack", "stages", "soft", "soft", "graph", "post"])
    if kind == "stack":
        par = rng.choice([dict(TUNED, margin=20), dict(EXAMPLE, margin=20), _draw_par(rng), _draw_par(rng)])
        W, H, L = _log_int(rng, 96, 2560), _log_int(rng, 96, 2160), _log_int(rng, 24, 160)
        L = max(24, min(L, int(1.6e8 / (W * H))))
        nuc = WIDE_NUCLEI if par["min_intensity"] == 1000 else NUCLEI
        return _stack(W, H, L, 32, rng.choice([1, 4, 8]), par, nuc, max(rng.uniform(2e-5, 1e-4), 100 / (W * H * L)), host=rng.random() < 0.5,
                      ave=rng.random() < 0.25)
    if kind == "stages":
        W, H, L = _log_int(rng, 64, 1280), _log_int(rng, 64, 1280), rng.randint(13, 40)
        return dict(kind="stages", W=W, H=H, L=L, density=max(rng.uniform(2e-5, 1e-4), 50 / (W * H * L)), erosion=rng.randint(1, 4), **_draw_par(rng), **NUCLEI)
    if kind == "soft":
        W, H, L = _log_int(rng, 40, 512), _log_int(rng, 40, 512), _log_int(rng, 14, 128)
        s = [round(rng.uniform(1.2, 2.6), 2), round(rng.uniform(1.2, 2.6), 2), round(rng.uniform(0.9, 1.8), 2)]
        points = max(16, min(4000, int(W * H * L * rng.choice([2e-5, 6e-5, 2e-4]))))
        return dict(kind="soft", W=W, H=H, L=L, rxy=_log_int(rng, 3, 40), rz=rng.randint(1, 6), points=points, keep=rng.random() < 0.75,
                    density=1e-4, sx1=s[0], sy1=s[1], sz1=s[2], sx2=round(1.6 * s[0], 2), sy2=round(1.6 * s[1], 2), sz2=round(1.6 * s[2], 2),
                    **NUCLEI)
    if kind == "graph":
        par = rng.choice([dict(TUNED, margin=10), dict(_draw_par(rng), margin=10)])
        return dict(kind="graph", W=rng.choice([128, 192, 256, 320]), H=rng.choice([96, 128, 256]), n=rng.randint(4, 16), depth=32, batch=16,
                    density=rng.uniform(5e-5, 1.2e-4), **par, **NUCLEI)
    return dict(kind="post", n=_log_int(rng, 1000, 1500000), ave=rng.random() < 0.5)


# ---------------------------------------------------------------- inputs
def _volume(c, W, H, L, seed):
    """uint16 (L, H, W) on the GPU and the nuclei's centres (n, 3) as z, y, x."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev = "cuda"
    n = max(4, int(round(c["density"] * W * H * L)))

    def uni(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device=dev)
    pos = torch.stack([uni(0, L - 1), uni(0, H - 1), uni(0, W - 1)], 1)
    sxy, sz, peak = uni(c["nxy_lo"], c["nxy_hi"]), uni(c["nz_lo"], c["nz_hi"]), uni(c["peak_lo"], c["peak_hi"])
    k = n // 20     # a tenth of the nuclei in touching pairs: k of them move next to k others
    ang = 2 * math.pi * torch.rand(k, generator=g, device=dev)
    dist = 0.8 * (sxy[:k] + sxy[k:2 * k])
    pos[k:2 * k] = pos[:k] + torch.stack([torch.zeros_like(ang), dist * torch.sin(ang), dist * torch.cos(ang)], 1)
    acc = torch.zeros(L * H * W, dtype=torch.int32, device=dev)   # sixteenths: an integer sum has one value
    ry, rz = int(math.ceil(2.8 * c["nxy_hi"])), int(math.ceil(2.8 * c["nz_hi"]))
    oz, oy, ox = torch.meshgrid(torch.arange(-rz, rz + 1, device=dev), torch.arange(-ry, ry + 1, device=dev),
                                torch.arange(-ry, ry + 1, device=dev), indexing="ij")
    off = torch.stack([oz, oy, ox], -1).reshape(1, -1, 3)
    step = max(1, 24_000_000 // off.shape[1])
    lim = torch.tensor([L, H, W], device=dev)
    for a in range(0, n, step):
        p = pos[a:a + step, None, :]
        q = p.round().to(torch.int64) + off
        d = q - p
        s2, z2 = sxy[a:a + step, None] ** 2, sz[a:a + step, None] ** 2
        v = peak[a:a + step, None] * torch.exp(-0.5 * ((d[..., 1] ** 2 + d[..., 2] ** 2) / s2 + d[..., 0] ** 2 / z2))
        ok = ((q >= 0) & (q < lim)).all(-1)
        acc.index_add_(0, ((q[..., 0] * H + q[..., 1]) * W + q[..., 2])[ok], (v[ok] * 16).to(torch.int32))
        del q, d, v, ok
    acc = acc.view(L, H, W)
    vol = torch.empty((L, H, W), dtype=torch.uint16, device=dev)
    for z in range(L):
        f = c["bg"] + c["bg_sd"] * torch.randn((H, W), generator=g, device=dev)
        f = f + acc[z] * ((1.0 - 0.4 * z / max(1, L - 1)) / 16)
        f = f * (1 + 0.05 * (2 * torch.rand((H, 1), generator=g, device=dev) - 1))
        vol[z] = f.round().clamp_(0, 65535).to(torch.int32).to(torch.uint16)
    return vol, pos


def _params(c, W, H, depth):
    m = min(c["margin"], W // 4, H // 4)
    return hdog.make_params(width=W, height=H, depth=depth, left_margin=m, right_margin=m, top_margin=m, bottom_margin=m,
                            extra_depth_margin=c["extra"], radius_norm_xy=c["rxy"], radius_norm_z=c["rz"],
                            min_intensity=c["min_intensity"], sigma_xy_small=c["sxy1"], sigma_z_small=c["sz1"],
                            sigma_xy_large=c["sxy2"], sigma_z_large=c["sz2"], min_size=c["min_size"],
                            is_ave_mode=int(c.get("ave", False)))


def _frames(c):
    """The graph case's stacks: (W, H, L) of each, uneven depths, full and half frames."""
    W, H = c["W"], c["H"]
    return [((W, H), (W // 2, H), (W, H // 2))[i % 3] + (64 + (i * 61) % 160,) for i in range(c["n"])]


def _records_array(c, voxels):
    """The program's own record array, kept across calls: a few times the blobs that noise at the small sigma leaves."""
    margin = _radius(c["sz2"]) + c["extra"]
    overlap = c["depth"] / max(1, c["depth"] - 2 * margin) if "depth" in c else 1.0
    return np.zeros(4000 + int(voxels * overlap * 0.015 / (c["sxy1"] ** 2 * c["sz1"])), hdog.DT_LOCAL)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "stack":
        vol, _ = _volume(c, c["W"], c["H"], c["L"], seed)
        ctx = hdog.Context(_params(c, c["W"], c["H"], c["depth"]), c["batch"])
        s = dict(kind=kind, ctx=ctx, out=_records_array(c, vol.numel()))
        if c["host"]:
            s["keep"] = torch.empty(vol.shape, dtype=torch.uint16, pin_memory=True)   # the program's own page-locked stack
            s["keep"].copy_(vol)
            s["stack"] = s["keep"].numpy()
        else:
            s["stack"] = vol
        return s
    if kind == "graph":
        frames = _frames(c)
        stacks = [_volume(c, w, h, n, seed * 100 + i)[0] for i, (w, h, n) in enumerate(frames)]
        ctxs = [hdog.Context(_params(c, w, h, c["depth"]), c["batch"]) for w, h in dict.fromkeys(f[:2] for f in frames)]
        return dict(kind=kind, graph=hdog.Graph(ctxs, stacks), out=_records_array(c, sum(v.numel() for v in stacks)))
    if kind == "stages":
        vol, _ = _volume(c, c["W"], c["H"], c["L"], seed)
        cap = len(_records_array(c, vol.numel()))
        table = {k: np.zeros((rows, cap), t) for k, rows, t in (("label", 1, np.int32), ("count", 1, np.uint32), ("intensity", 1, np.float32),
                                                                ("centroid", 3, np.float32), ("hessian", 6, np.float32), ("eigen", 2, np.float32))}
        return dict(kind=kind, ctx=hdog.Context(_params(c, c["W"], c["H"], c["L"])), vol=vol, erosion=c["erosion"], table=table)
    if kind == "soft":
        vol, nuc = _volume(c, c["W"], c["H"], c["L"], seed)
        lim = torch.tensor([c["L"] - 1, c["H"] - 1, c["W"] - 1], device="cuda")
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 1)
        n = c["points"]
        pick = torch.randint(0, nuc.shape[0], (n,), generator=g, device="cuda")
        pos = (nuc[pick] + torch.rand((n, 3), generator=g, device="cuda") - 0.5).round()
        neg = torch.rand((n, 3), generator=g, device="cuda") * (lim + 1)
        vol = vol.to(torch.float32).requires_grad_(True)
        sigma = torch.tensor([c[k] for k in ("sx1", "sy1", "sz1", "sx2", "sy2", "sz2")], requires_grad=True)
        return dict(kind=kind, vol=vol, sigma=sigma, thresh=torch.zeros(3, requires_grad=True),
                    pos=torch.minimum(pos.clamp(min=0), lim).to(torch.int32), neg=torch.minimum(neg.floor(), lim).to(torch.int32),
                    kw=dict(radius_norm_xy=c["rxy"], radius_norm_z=c["rz"], min_intensity=50.0, tau=0.02, keep_intermediates=c["keep"]))
    rng = np.random.default_rng(seed)
    rec = np.zeros(c["n"], hdog.DT_LOCAL)
    for f, lo, hi in (("local_x", 0, 2560), ("local_y", 0, 2160), ("local_z", 0, 128)):
        rec[f] = rng.uniform(lo, hi, c["n"])
    for f, mu in (("structureness", -4.0), ("blobness", -1.0), ("intensity", 0.0)):
        rec[f] = np.exp(rng.normal(mu, 1.0, c["n"]))
    rec["size"] = rng.integers(1, 900, c["n"])
    return dict(kind=kind, rec=rec, ave=c["ave"], rng=None)


# ---------------------------------------------------------------- one pass
_GLOBAL = dict(offset=(10400.0, 8200.5, 312.25), scales=(1.3, -1.3, 5.0), image_size=(2560, 2160), i_xy=(3, 4))
_MERGE = dict(bound_z=(400.0, 880.0), margin_left=12, margin_top=8, offset=(9000.0, 4000.0, 100.0), coeff=(0.02, 0.02, 0.1),
              A=((0, 1, 0), (-1, 0, 0), (0, 0, 1)), b=(5.0, 900.0, 0.0))
_CLF = dict(bias=(0.5, 2.0, 1.0), scale=(1.0, 0.5, 2.0), bias_before_log=(0.0, 1e-6, 1e-6))


def _fields(r):
    return {f: r[f] for f in r.dtype.names}


def _found(out, rec):
    """The record array and how many of it the call filled; beyond them it is as it was."""
    assert len(rec) <= len(out), "the record array is too small"
    return dict(_fields(out), n=len(rec))


def run(state):
    kind = state["kind"]
    if kind == "stack":
        return _found(state["out"], state["ctx"].run_stack(state["stack"], out=state["out"]))
    if kind == "graph":
        rec, counts = state["graph"].run(out=state["out"])
        return dict(_found(state["out"], rec), counts=counts)
    if kind == "stages":
        ctx, vol = state["ctx"], state["vol"]
        ero = ctx.erosion(vol, state["erosion"], 1)
        norm = ctx.normalize(vol)
        dog = ctx.dog(norm)
        mask, hess = ctx.hessian_pd(dog, want_hessian=True)
        labels = ctx.ccl(mask)
        r, table = ctx.regional_features(labels, norm, dog), state["table"]
        for k, a in table.items():
            a[:, :r["num_regions"]] = r[k]
        return dict(erosion=ero.view(torch.int16), norm=norm, dog=dog, mask=mask, hess=hess, labels=labels, regions=table,
                    num_regions=r["num_regions"])
    if kind == "soft":
        loss = hdog.soft.soft_loss(state["vol"], state["sigma"], state["pos"], state["neg"], thresh=state["thresh"], **state["kw"])
        gv, gs, gb = torch.autograd.grad(loss, (state["vol"], state["sigma"], state["thresh"]))
        return dict(loss=loss.detach(), grad_volume=gv, grad_sigma=gs, grad_thresh=gb)
    g = hdog.records_to_global(state["rec"], is_fw=True, **_GLOBAL)
    m = hdog.scale_merge(g, **_MERGE)
    x = hdog.classifier_features(state["rec"], is_ave=state["ave"], **_CLF)
    return dict(merged=_fields(g), scaled=_fields(m), features=x)


# ---------------------------------------------------------------- what a pass cannot do without
def _radius(s):
    return int(2.0 * s + 0.5)


def _detect_flops(c):
    """Per processed voxel: the box sums of both extremes, the taps of both scales, the Hessian and its test."""
    taps = sum(2 * (2 * _radius(c["sxy%d" % i]) + 1) + 2 * _radius(c["sz%d" % i]) + 1 for i in (1, 2))
    return 2 * (2 * (2 * c["rxy"] + 1) + 2 * c["rz"] + 1) + 2 * taps + 50


def _substacks(L, depth, c):
    margin = _radius(c["sz2"]) + c["extra"]
    return len(hdog.substack_schedule(L, depth, margin))


def work(case):
    c, kind = case, case["kind"]
    if kind == "stack":
        n, subs = c["W"] * c["H"] * c["L"], _substacks(c["L"], c["depth"], c)
        return dict(bytes=2 * n + 28 * c["density"] * n, flops=c["W"] * c["H"] * c["depth"] * subs * _detect_flops(c))
    if kind == "graph":
        n = sum(w * h * k for w, h, k in _frames(c))
        done = sum(w * h * c["depth"] * _substacks(k, c["depth"], c) for w, h, k in _frames(c))
        return dict(bytes=2 * n + 28 * c["density"] * n, flops=done * _detect_flops(c))
    if kind == "stages":   # erosion 2 + 2, normalize 2 + 4, DoG 4 + 4, Hessian 4 + 25, labels 1 + 4, features 12
        n = c["W"] * c["H"] * c["L"]
        return dict(bytes=64 * n, flops=n * _detect_flops(c))
    if kind == "soft":     # the volume in, its gradient out
        n = c["W"] * c["H"] * c["L"]
        return dict(bytes=8 * n, flops=n * 8 * (2 * (2 * c["rxy"] + 1) + 2 * c["rz"] + 1))
    return dict(bytes=c["n"] * (28 + 15 + 15 + 13 + 28 + 24), flops=c["n"] * 60)


# ---------------------------------------------------------------- the same outputs in 64 bits
def _shift(x, axis, k):
    """x[i + k] along `axis`, zero outside."""
    n = x.shape[axis]
    y = torch.zeros_like(x)
    if abs(k) < n:
        y.narrow(axis, max(0, -k), n - abs(k)).copy_(x.narrow(axis, max(0, k), n - abs(k)))
    return y


def _clamped(x, axis, r):
    n = x.shape[axis]
    return x.index_select(axis, torch.arange(-r, n + r, device=x.device).clamp(0, n - 1))


def _extreme(x, axis, r, is_max):
    p = _clamped(x, axis, r)
    span, f = 1, torch.maximum if is_max else torch.minimum
    while 2 * span <= 2 * r + 1:
        p = f(p.narrow(axis, 0, p.shape[axis] - span), p.narrow(axis, span, p.shape[axis] - span))
        span *= 2
    return f(p.narrow(axis, 0, x.shape[axis]), p.narrow(axis, 2 * r + 1 - span, x.shape[axis]))


def _box(x, axis, r):
    p = _clamped(x, axis, r).cumsum(axis)
    z = torch.zeros_like(p.narrow(axis, 0, 1))
    p = torch.cat([z, p], axis)
    n = x.shape[axis]
    return (p.narrow(axis, 2 * r + 1, n) - p.narrow(axis, 0, n)) / (2 * r + 1)


def _normalized(vol, rxy, rz, min_intensity):
    means = []
    for is_max in (False, True):
        e = vol
        for axis, r in ((2, rxy), (1, rxy), (0, rz)):
            e = _extreme(e, axis, r, is_max)
        for axis, r in ((2, rxy), (1, rxy), (0, rz)):
            e = _box(e, axis, r)
        means.append(e)
    return torch.where(vol >= min_intensity, (vol - means[0]) / (means[1] - means[0]), torch.zeros_like(vol))


def _taps(s):
    r = _radius(float(s))
    k = torch.arange(-r, r + 1, dtype=torch.float64, device="cuda")
    t = torch.exp(-0.5 * k * k / (s * s))
    return t / t.sum()


def _conv(x, axis, t):
    r = (t.numel() - 1) // 2
    y = torch.zeros_like(x)
    for k in range(-r, r + 1):
        y = y + t[k + r] * _shift(x, axis, k)
    return y


def _smooth(x, sx, sy, sz):
    return _conv(_conv(_conv(x, 2, _taps(sx)), 1, _taps(sy)), 0, _taps(sz))


def _hessian(f):
    g = [0.5 * (_shift(f, a, 1) - _shift(f, a, -1)) for a in (2, 1, 0)]
    return [0.5 * (_shift(g[i], a, 1) - _shift(g[i], a, -1)) for i, a in ((0, 2), (0, 1), (0, 0), (1, 1), (1, 0), (2, 0))]


def _soft_points(norm, p, sigma, thresh, tau):
    """The relaxed mask score at the points: the separable Gaussians, evaluated on the points' own
    neighbourhoods (with the volume's zero borders), then the Hessian's differences and the test."""
    reach = [max(_radius(float(sigma[i])), _radius(float(sigma[i + 3]))) for i in (2, 1, 0)]   # z, y, x
    at = [p[:, a, None] + torch.arange(-reach[a] - 2, reach[a] + 3, device=p.device) for a in range(3)]
    inside = [(at[a] >= 0) & (at[a] < norm.shape[a]) for a in range(3)]
    i = [at[a].clamp(0, norm.shape[a] - 1) for a in range(3)]
    v = norm[i[0][:, :, None, None], i[1][:, None, :, None], i[2][:, None, None, :]]
    v = v * (inside[0][:, :, None, None] & inside[1][:, None, :, None] & inside[2][:, None, None, :])
    dog = 0
    for k, sign in ((0, 1.0), (3, -1.0)):
        u = v
        for axis, s in ((3, sigma[k]), (2, sigma[k + 1]), (1, sigma[k + 2])):
            t = _taps(s)
            r, h = (t.numel() - 1) // 2, reach[axis - 1]
            u = sum(t[j + r] * u.narrow(axis, h + j, 5) for j in range(-r, r + 1))
        dog = dog + sign * u
    live = [m[:, reach[a]:reach[a] + 5].to(torch.float64) for a, m in enumerate(inside)]   # zero outside the volume
    live = live[0][:, :, None, None] * live[1][:, None, :, None] * live[2][:, None, None, :]
    dog = dog * live * (sigma[0] * sigma[1] * sigma[2])

    def diff(f, axis, m):   # central difference at the inner positions, zero where the position is outside
        n = f.shape[axis]
        return 0.5 * (f.narrow(axis, 2, n - 2) - f.narrow(axis, 0, n - 2)) * m.narrow(axis, 1, n - 2)
    h = []
    for a, b in ((3, 3), (3, 2), (3, 1), (2, 2), (2, 1), (1, 1)):
        g = diff(dog, a, live)
        gl = live.narrow(a, 1, 3)
        g = diff(g, b, gl)
        h.append(g[:, g.shape[1] // 2, g.shape[2] // 2, g.shape[3] // 2])
    xx, xy, xz, yy, yz, zz = h
    det = xx * yy * zz + 2 * xy * yz * xz - xx * yz * yz - yy * xz * xz - zz * xy * xy
    return torch.sigmoid((thresh[0] - xx) / tau) * torch.sigmoid((xx * yy - xy * xy - thresh[1]) / tau ** 2) * \
        torch.sigmoid((thresh[2] - det) / tau ** 3)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "stages":
        vol, _ = _volume(c, c["W"], c["H"], c["L"], seed)
        f32 = {k: float(np.float32(c[k])) for k in ("sxy1", "sz1", "sxy2", "sz2")}
        norm = _normalized(vol.to(torch.float64), c["rxy"], c["rz"], c["min_intensity"])
        dog = (_smooth(norm, f32["sxy1"], f32["sxy1"], f32["sz1"]) - _smooth(norm, f32["sxy2"], f32["sxy2"], f32["sz2"])) * \
            (f32["sxy1"] ** 2 * f32["sz1"])
        return dict(erosion=None, norm=norm, dog=dog, mask=None, hess=torch.stack(_hessian(dog)), labels=None, regions=None,
                    num_regions=None)
    if kind == "soft":   # the volume's gradient has no such value: which of several equal extremes it goes to is a choice
        s = prepare(case, seed)
        norm = _normalized(s["vol"].detach().to(torch.float64), c["rxy"], c["rz"], 50.0)
        sigma = s["sigma"].detach().to(torch.float64).cuda().requires_grad_(True)
        thresh = torch.zeros(3, dtype=torch.float64, device="cuda", requires_grad=True)
        loss = 0.0
        gs, gb = torch.zeros(6, dtype=torch.float64, device="cuda"), torch.zeros(3, dtype=torch.float64, device="cuda")
        for p, sign in ((s["pos"], 1.0), (s["neg"], -1.0)):
            for q in p.split(256):
                part = sign * _soft_points(norm, q.to(torch.int64), sigma, thresh, 0.02).sum() / p.shape[0]
                a, b = torch.autograd.grad(part, (sigma, thresh))
                gs, gb, loss = gs + a, gb + b, loss + part.detach()
        return dict(loss=loss, grad_volume=None, grad_sigma=gs, grad_thresh=gb)
    if kind == "post":
        r = prepare(case, seed)["rec"]
        f = {k: r[k].astype(np.float64) for k in r.dtype.names}
        o, s, size = _GLOBAL["offset"], _GLOBAL["scales"], _GLOBAL["image_size"]
        m = [o[a] + f["local_" + "xyz"[a]] * s[a] - (size[a] * s[a] if a < 2 and s[a] < 0 else 0) for a in range(3)]
        k = np.stack([(m[a] - _MERGE["offset"][a]) * _MERGE["coeff"][a] - (_MERGE["margin_left"], _MERGE["margin_top"], 0)[a] for a in range(3)])
        w = np.array(_MERGE["A"], np.float64) @ k + np.array(_MERGE["b"])[:, None]
        first = f["intensity"] / f["size"] if c["ave"] else f["intensity"]
        F = np.stack([first, f["structureness"], f["blobness"]], 1)
        x = (np.log10(F + np.array(_CLF["bias_before_log"])) + np.array(_CLF["bias"])) * np.array(_CLF["scale"])
        return dict(merged=dict(merged_x=m[0], merged_y=m[1], merged_z=m[2], i_x=None, i_y=None, FWRV=None),
                    scaled=dict(scaled_x=w[0], scaled_y=w[1], scaled_z=w[2], is_valid=None), features=x)
    return None
