"""A graph that mixes contexts whose batches run one after the other (2^28 voxels and more, here two substacks of
2048 x 2048 x 32) with contexts whose batches run beside them: the records of the plain per-stack calls, byte for byte."""
import numpy as np
import pytest
import torch

from helpers import params

SHAPES = [(2048, 2048), (128, 96), (96, 64)]


@pytest.mark.gpu
def test_gpu_graph_of_large_and_small_batches():
    import hdog
    p_of = lambda W, H: params(W, H, 32, margins=4)
    gen = torch.Generator(device="cuda").manual_seed(5)
    dev = []
    for i, (W, H) in enumerate(SHAPES + SHAPES[1:] + SHAPES[:1]):
        v = torch.randint(90, 130, (40 + 7 * i, H, W), generator=gen, device="cuda", dtype=torch.int32)
        at = torch.randint(0, v.numel(), (v.numel() // 20000 + 20,), generator=gen, device="cuda")
        v.view(-1)[at] = 4000
        dev.append(v.to(torch.uint16))
    recs = []
    for v in dev:
        with hdog.Context(p_of(v.shape[2], v.shape[1]), max_substacks=1) as ctx:
            recs.append(ctx.run_stack(v))
    ctxs = [hdog.Context(p_of(w, h), max_substacks=2) for w, h in SHAPES]
    with hdog.Graph(ctxs, dev) as g:
        for _ in range(2):
            got, counts = g.run()
            assert list(counts) == [len(r) for r in recs] and min(counts) > 0
            assert got.tobytes() == np.concatenate(recs).tobytes()
    for c in ctxs:
        c.close()
