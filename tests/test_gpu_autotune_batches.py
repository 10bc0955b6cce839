"""The autotuner's choice belongs to what it was timed on: the substacks of the batch, and whether the sweeps ran.
A graph of many substacks does not take the launch shapes and the batch that a graph of one left behind."""
import numpy as np
import pytest
import torch

from helpers import params, volume

pytestmark = pytest.mark.gpu


def frames(W, H, seed):
    one = torch.from_numpy(volume(W, H, 24, seed=seed)).cuda()     # one substack
    many = torch.from_numpy(volume(W, H, 150, seed=seed + 1)).cuda()
    return one, many


def p_of(W, H):
    return params(W, H, 32, margins=4)


def graph(hdog, ctx, v, ref):
    with hdog.Graph([ctx], [v]) as g:
        got, _ = g.run()
    assert got.tobytes() == ref.tobytes()
    return ctx.tuning()


@pytest.mark.parametrize("same_context", [False, True])
def test_gpu_a_graph_is_tuned_on_its_own_batch(same_context):
    import hdog
    W, H = (176, 112) if same_context else (176, 120)
    one, many = frames(W, H, 301)
    with hdog.Context(p_of(W, H)) as c:
        refs = [c.run_stack(v) for v in (one, many)]
    a = hdog.Context(p_of(W, H), max_substacks=4)
    b = a if same_context else hdog.Context(p_of(W, H), max_substacks=4)
    assert graph(hdog, a, one, refs[0])["tuned_on_substacks"] == 1
    t = graph(hdog, b, many, refs[1])
    assert t["tuned_on_substacks"] == 4 and t["batch"] in (2, 4), t
    # the same batch again: the kept timings, not new ones
    assert graph(hdog, b, many, refs[1]) == t
    with hdog.Context(p_of(W, H), max_substacks=4) as d:
        assert graph(hdog, d, many, refs[1]) == t
    a.close()
    b.close()


def test_gpu_tuning_without_the_sweeps_is_not_kept_for_them():
    import hdog
    W, H = 176, 104
    _, many = frames(W, H, 311)
    with hdog.Context(p_of(W, H)) as c:
        ref = c.run_stack(many)
    with hdog.Context(p_of(W, H), max_substacks=4) as c:
        c.set_fused_sweep(False)
        assert graph(hdog, c, many, ref)["k_hess_sweep_ms"] == [0, 0, 0]
    with hdog.Context(p_of(W, H), max_substacks=4) as c:
        assert np.all(np.array(graph(hdog, c, many, ref)["k_hess_sweep_ms"]) > 0)
