"""Gather and scatter-add for row lengths of every access width, narrow rows, and few ids (sorted by one CTA): sizes at
the edges, against the oracle."""
import numpy as np
import pytest

import gpu_util as G
from conftest import assert_close
from oracle import fused_layers as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,C,n", [(7, 1, 1), (50, 3, 64), (300, 33, 65), (5000, 129, 4096), (5000, 130, 4097), (100, 64, 2049),
                                   (70000, 45, 9000), (151936, 694, 3000), (65, 514, 60000), (640, 128, 192), (2, 20, 4000)])
def test_gather_and_scatter_add(V, C, n):
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(V + C + n)
    ids_ = np.minimum((V * rng.random(n) ** 3).astype(np.int32), V - 1)   # hot rows
    table_ = rng.standard_normal((V, C), dtype=np.float32)
    dout_ = rng.standard_normal((n, C), dtype=np.float32)
    grad_ = rng.standard_normal((V, C), dtype=np.float32)
    ids, table = G.up(ids_, requires_grad=False), G.up(table_, grad=grad_)
    out = G.empty((n, C), grad=dout_)
    node = G.node("GatherOp", (ids, table), (out,))
    G.run_forward(node)
    assert np.array_equal(G.down(out), table_[ids_])
    G.run_backward(node)
    ref = grad_.astype(np.float64)
    np.add.at(ref, ids_, dout_.astype(np.float64))
    got = G.down(table.grad)
    count = np.bincount(ids_, minlength=V)
    scale = np.sqrt(1.0 + count)[:, None]
    assert np.abs((got - ref) / scale).max() < 1e-5
    assert np.array_equal(got[count == 0], grad_[count == 0])
    once = count == 1
    seq = grad_.copy()
    np.add.at(seq, ids_, dout_)
    assert np.array_equal(got[once], seq[once])
    be.copy_from_host(table.grad, grad_)
    G.run_backward(node)
    assert np.array_equal(G.down(table.grad), got)      # the same bits again
    bits = G.bf16_grad(table, O.f32_to_bf16_bits(grad_))
    G.run_backward(node)
    want = O.round_to_bf16(grad_).astype(np.float64)
    np.add.at(want, ids_, dout_.astype(np.float64))
    assert_close(O.bf16_bits_to_f32(G.down_bits(bits)) / scale, want / scale, 1e-2, "bf16 table gradient")
    G.check_clean_status()


def test_bad_ids_in_a_short_list():
    ctx, alloc, be = G.env()
    ids_ = np.array([3, -1, 3, 9, 10, 2**31 - 1], np.int32)
    ids, table = G.up(ids_, requires_grad=False), G.up(np.zeros((10, 6), np.float32), grad=0)
    out = G.empty((6, 6), grad=np.ones((6, 6), np.float32))
    G.run_backward(G.node("GatherOp", (ids, table), (out,)))
    got = G.down(table.grad)
    assert got[3].tolist() == [2.0] * 6 and got[9].tolist() == [1.0] * 6 and got.sum() == 18.0
    assert ctx.status() == 1
