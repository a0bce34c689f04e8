"""Scatter-add of very few ids, which one launch does without a sort: rows of every number of pieces and access width, one id for
all positions, the largest list of this kind and the smallest of the next, against the oracle."""
import numpy as np
import pytest

import gpu_util as G
import test_gpu_embed_widths as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,C,n", [(1, 128, 512), (1, 257, 33), (2, 514, 511), (65, 384, 512), (65, 512, 300), (9, 640, 31), (9, 1280, 32),
                                   (3000, 4100, 100), (65, 2049, 257), (40, 66, 513), (1, 5, 1024), (3, 100, 1025), (3, 512, 1024),
                                   (3, 1300, 256), (3, 516, 257)])
def test_gather_and_scatter_add(V, C, n):
    W.test_gather_and_scatter_add(V, C, n)


@pytest.mark.parametrize("C", [36, 640])
def test_short_segments_are_added_in_order(C):
    """A row whose occurrences one warp adds: the bits of adding them one after the other (rows of five pieces and more)."""
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(C)
    ids_ = rng.integers(0, 40, 200).astype(np.int32)
    dout_, grad_ = rng.standard_normal((200, C), dtype=np.float32), rng.standard_normal((40, C), dtype=np.float32)
    ids, table = G.up(ids_, requires_grad=False), G.up(np.zeros((40, C), np.float32), grad=grad_)
    out = G.empty((200, C), grad=dout_)
    G.run_backward(G.node("GatherOp", (ids, table), (out,)))
    want = grad_.copy()
    np.add.at(want, ids_, dout_)
    got = G.down(table.grad)
    if C >= 5 * 128:
        assert np.array_equal(got, want)
    else:
        assert np.abs(got - want).max() < 1e-5
    G.check_clean_status()
    G.free(ids, table, out)


@pytest.mark.parametrize("C", [36, 130, 257, 384, 514, 1283, 2600])
def test_up_to_sixteen_occurrences_are_added_in_order(C):
    """Whatever the row length and the other ids, the bits of adding them one after the other onto the row."""
    rng = np.random.default_rng(C)
    ids_ = rng.permutation(np.repeat(np.arange(16), np.arange(1, 17))).astype(np.int32)
    n = len(ids_)
    dout_, grad_ = rng.standard_normal((n, C), dtype=np.float32), rng.standard_normal((20, C), dtype=np.float32)
    ids, table = G.up(ids_, requires_grad=False), G.up(np.zeros((20, C), np.float32), grad=grad_)
    out = G.empty((n, C), grad=dout_)
    G.run_backward(G.node("GatherOp", (ids, table), (out,)))
    want = grad_.copy()
    np.add.at(want, ids_, dout_)
    assert np.array_equal(G.down(table.grad), want)
    G.check_clean_status()
    G.free(ids, table, out)


@pytest.mark.parametrize("pattern", ["one", "half", "two", "seventeen"])
@pytest.mark.parametrize("n,C", [(1024, 512), (1024, 36), (1023, 130), (1000, 257), (256, 1283), (256, 5000), (40, 2600), (250, 4096)])
def test_frequent_ids(n, C, pattern):
    """Ids that many or all positions name, as in a padded batch: their blocks share the pieces of the row, their warps the
    positions.  A sum of k terms errs by k 2^-24 of their sizes at most; the same bits in every run."""
    rng = np.random.default_rng(n + C)
    ids_ = {"one": np.full(n, 7), "half": np.where(np.arange(n) % 2, 3, rng.integers(0, 50, n)), "two": np.arange(n) % 2,
            "seventeen": np.arange(n) // 17}[pattern].astype(np.int32)
    V = int(ids_.max()) + 2
    dout_, grad_ = rng.standard_normal((n, C), dtype=np.float32), rng.standard_normal((V, C), dtype=np.float32)
    ids, table = G.up(ids_, requires_grad=False), G.up(np.zeros((V, C), np.float32), grad=grad_)
    out = G.empty((n, C), grad=dout_)
    node = G.node("GatherOp", (ids, table), (out,))
    ctx, alloc, be = G.env()
    runs = []
    for _ in range(2):
        be.copy_from_host(table.grad, grad_)
        G.run_backward(node)
        runs.append(G.down(table.grad))
    assert np.array_equal(runs[0], runs[1])
    want, size = grad_.astype(np.float64), np.abs(grad_).astype(np.float64)
    np.add.at(want, ids_, dout_.astype(np.float64))
    np.add.at(size, ids_, np.abs(dout_).astype(np.float64))
    terms = 1 + np.bincount(ids_, minlength=V)[:, None]
    assert (np.abs(runs[0] - want) <= terms * 2.0 ** -24 * size).all()
    G.check_clean_status()
    G.free(ids, table, out)


def test_a_frequent_id_costs_little_more_than_distinct_ones():
    """One id for all positions within four times the time of as many different ids (it is twice; one block walking all the
    positions makes it ten times)."""
    ctx, alloc, be = G.env()
    n, C = 256, 1280
    table = G.up(np.zeros((n, C), np.float32), grad=0)
    out = G.empty((n, C), grad=np.ones((n, C), np.float32))
    nbytes = ctx.scatter_add_scratch_bytes(n, C, n)
    scratch = G.empty((nbytes // 4 + 1,))
    us = []
    for ids_ in (np.arange(n), np.full(n, 5)):
        ids = G.up(ids_.astype(np.int32), requires_grad=False)
        args = (ids.storage.ptr.address, out.grad.storage.ptr.address, table.grad.storage.ptr.address, scratch.storage.ptr.address,
                nbytes, n, C, n)
        ctx.gather_backward(*args)
        ctx.synchronize()
        g = ctx.record(lambda r: [r.gather_backward(*args) for _ in range(20)])
        times = []
        for _ in range(9):
            ctx.event_record(0)
            ctx.replay(g)
            ctx.event_record(1)
            times.append(ctx.event_elapsed_ms(0, 1) * 50)
        ctx.drop_recording(g)
        us.append(sorted(times)[4])
        G.free(ids)
    print("%d x %d: distinct %.1f us, one id %.1f us" % (n, C, *us))
    assert us[1] < 4 * us[0]
    G.free(table, out, scratch)
