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
