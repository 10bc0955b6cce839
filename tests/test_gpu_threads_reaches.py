"""Calls with different window reaches side by side on several host threads (csrc/soft.cu, csrc/norm.cu): the reaches need
different amounts of shared memory above 48 KB from the same kernels, and no call may take another's
allowance away between setting it and its launch.  Each thread works on its own stream and buffers."""
import ctypes
import threading

import numpy as np
import pytest
import torch

ROUNDS = 1500


def side_by_side(calls):
    errors, start = [], threading.Barrier(len(calls))

    def work(f):
        start.wait()
        try:
            for _ in range(ROUNDS):
                f()
        except Exception as e:   # reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(f,)) for f in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors


@pytest.mark.gpu
def test_gpu_soft_calls_with_different_reaches_on_several_threads():
    import hdog
    from hdog.soft import _params
    L = hdog.lib()
    q = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    vol = torch.tensor(np.random.default_rng(2).uniform(100, 900, (12, 40, 48)).astype(np.float32), device="cuda")
    pos = torch.tensor([[5, 20, 20], [6, 30, 40]], dtype=torch.int32, device="cuda")
    neg = torch.tensor([[2, 3, 4]], dtype=torch.int32, device="cuda")
    keep = []

    def call(r):
        prm = _params(vol, torch.tensor([1.0, 1.0, 1.0, 1.6, 1.6, 1.6]), torch.zeros(3), (r, 2, 50.0, 0.05, 1.0))
        st = torch.cuda.Stream()
        ws = torch.empty(L.hdog_soft_workspace_bytes(ctypes.byref(prm)), dtype=torch.uint8, device="cuda")
        loss, gv, gs, gb = (torch.empty(n, device="cuda") for n in (1, vol.numel(), 6, 3))
        keep.append((prm, st, ws, loss, gv, gs, gb))
        s = ctypes.c_void_p(st.cuda_stream)

        def f():
            hdog.check(L.hdog_soft_forward(ctypes.byref(prm), q(vol), q(pos), 2, q(neg), 1, q(loss), None, q(ws), s))
            hdog.check(L.hdog_soft_backward_kept(ctypes.byref(prm), q(vol), q(pos), 2, q(neg), 1, 1.0, q(gv), q(gs), q(gb),
                                                 q(ws), s))
        return f

    torch.cuda.synchronize()
    side_by_side([call(40), call(100), call(340)])


@pytest.mark.gpu
def test_gpu_contexts_with_different_reaches_on_several_threads():
    import hdog
    rng = np.random.default_rng(3)
    vol = torch.from_numpy(rng.integers(100, 4000, (4, 48, 64)).astype(np.uint16)).cuda()
    ctxs = [hdog.Context(hdog.make_params(width=64, height=48, depth=4, radius_norm_xy=r, radius_norm_z=2))
            for r in (90, 300, 400, 300, 200, 421)]
    want = [c.normalize(vol).cpu() for c in ctxs]
    streams = [torch.cuda.Stream() for _ in ctxs]
    torch.cuda.synchronize()
    side_by_side([lambda c=c, s=s: c.normalize(vol, stream=s) for c, s in zip(ctxs, streams)])
    assert all(torch.equal(c.normalize(vol).cpu(), w) for c, w in zip(ctxs, want))
    for c in ctxs:
        c.close()
