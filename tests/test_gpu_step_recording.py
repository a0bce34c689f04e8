"""A step that replays its recorded launches gives the bits of the launches made one by one, counts them alike, follows
a changed descriptor, and steps aside for event timing and for a program that captures the stream itself."""
import numpy as np
import pytest
import torch

import autograd_b200 as ag
import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu

BATCHES = 6


def _step(env, n_layer):
    from autograd_b200.step import FusedLayerStep, StepConfig
    cfg = StepConfig(n_layer=n_layer, n_embd=128, n_head=1, head_dim=128, seq_len=40, vocab=392, batch=3)
    rng = np.random.default_rng(n_layer)
    return FusedLayerStep(*env, cfg, seed=9), rng.integers(0, 392, (BATCHES, 2, 120)).astype(np.int32)


def _load(ctx, st, batch):
    ctx.copy_from_host(st.ids, batch[0])
    ctx.copy_from_host(st.targets, batch[1])


def _results(ctx, st):
    shapes = ((st.small_bucket, st.n_small + 1), (st.dtable, st.V * st.C), (st.dh, st.N * st.C), (st.q, st.N * st.C))
    return [ctx.copy_to_host(a, (n,), np.uint32).copy() for a, n in shapes]


@pytest.mark.parametrize("n_layer", [0, 2])
def test_replayed_step_equals_launched_step(n_layer):
    env = G.env()
    ctx = env[0]
    one, batches = _step(env, n_layer)
    two, _ = _step(env, n_layer)
    for i, b in enumerate(batches):
        counts = []
        two.timer.enabled = i == 3
        for st in (one, two):
            if i == 4:      # another descriptor: what was recorded with the first one is not replayed
                st.desc = ctx.flce_desc(st.N, st.C, st.V, vocab_chunk=st.cfg.ce_vocab_chunk, precision=N.AG_CE_BF16X3)
            _load(ctx, st, b)
            c0 = ctx.launch_count
            if st is one:
                st.forward()
                st.backward()
            else:
                st.step()
            counts.append(ctx.launch_count - c0)
        assert counts[0] == counts[1]
        for x, y in zip(_results(ctx, one), _results(ctx, two)):
            np.testing.assert_array_equal(x, y)
    assert two._graph is not None
    G.check_clean_status()
    one.close()
    two.close()


@pytest.mark.parametrize("warm_up", [1, 2])
def test_capture_after_few_steps(warm_up):
    """A program that warms up with one step and captures the next: the launches of that step are in its graph, and the
    step itself records nothing until the capture is over."""
    stream = torch.cuda.Stream()
    ctx = ag.context.CudaContext(0, stream.cuda_stream)
    st, batches = _step((ctx, G.env()[1], G.env()[2]), 1)
    _load(ctx, st, batches[0])
    for _ in range(warm_up):
        st.step()
    before = st._graph
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        st.step()
    assert st._graph == before
    with torch.cuda.stream(stream):
        graph.replay()
    got = _results(ctx, st)[:3]
    st.forward()
    st.backward()
    for x, y in zip(got, _results(ctx, st)[:3]):
        np.testing.assert_array_equal(x, y)
    st.step()
    st.step()
    assert st._graph is not None
    st.close()
    ctx.close()


def test_step_inside_a_captured_stream():
    stream = torch.cuda.Stream()
    ctx = ag.context.CudaContext(0, stream.cuda_stream)
    alloc = G.env()[1]
    st, batches = _step((ctx, alloc, G.env()[2]), 1)
    for b in batches[:3]:
        _load(ctx, st, b)
        st.step()
    want = _results(ctx, st)[:3]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        st.step()
    ctx.fill_f32(st.dtable, 7.0, st.V * st.C)
    with torch.cuda.stream(stream):
        graph.replay()
    for x, y in zip(want, _results(ctx, st)[:3]):
        np.testing.assert_array_equal(x, y)
    st.close()
    ctx.close()
