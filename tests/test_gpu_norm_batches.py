"""Norms whose dgamma and dbeta are added up together, against each by itself, bit for bit; and three ranges cleared at once."""
import ctypes

import numpy as np
import pytest
import torch

import gpu_util as G
from autograd_b200 import AgError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norms,n,c", [(1, 5, 128), (3, 192, 128), (64, 40, 36), (65, 33, 130), (2, 9000, 128), (2, 700, 2052)])
def test_partial_rows_added_together(norms, n, c):
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    dy, x, res = (torch.randn(norms, n, c, device="cuda", generator=g) for _ in range(3))
    gamma = torch.randn(norms, c, device="cuda", generator=g)
    one, two = torch.randn(norms, 2, c, device="cuda", generator=g), None
    two = one.clone()
    dx, dx2 = torch.empty_like(x), torch.empty_like(x)
    nbytes = ctx.norm_partials_bytes(c)
    part = torch.empty(norms, nbytes // 4, device="cuda")
    rows = (ctypes.c_int32 * norms)()
    torch.cuda.synchronize()
    for i in range(norms):
        a = [t[i].data_ptr() for t in (dy, x, gamma, res)]
        ctx.layernorm_backward(*a, dx[i].data_ptr(), one[i, 0].data_ptr(), one[i, 1].data_ptr(), part.data_ptr(), nbytes, n, c,
                               1e-5)
    ctx.synchronize()
    for i in range(norms):
        a = [t[i].data_ptr() for t in (dy, x, gamma, res)]
        ctx.layernorm_backward_rows(*a, dx2[i].data_ptr(), part[i].data_ptr(), nbytes, ctypes.addressof(rows) + 4 * i, n, c, 1e-5)
    ctx.norm_partials_add(part.data_ptr(), nbytes // 4, ctypes.addressof(rows), norms, c, two.data_ptr())
    ctx.synchronize()
    G.check_clean_status()
    assert min(rows) > 0 and torch.equal(dx, dx2)
    # beyond 512 partial rows the launch of one norm adds them in another order: n terms, half an ulp of their sizes each at worst
    if max(rows) <= 512:
        assert torch.equal(one, two)
    else:
        bound = n * 2.0 ** -24 * dy.abs().sum(1).max()
        assert float((one - two).abs().max()) <= 8 * float(bound)
    rows[0] = nbytes // (8 * c) + 1
    if norms > 1:
        with pytest.raises(AgError):
            ctx.norm_partials_add(part.data_ptr(), nbytes // 4, ctypes.addressof(rows), norms, c, two.data_ptr())


@pytest.mark.parametrize("sizes", [(1, 0, 0), (5, 3, 1026), (0, 70000, 7), ((1 << 24) - 8, 4, 4), (1 << 23, 1 << 23, 1)])
@pytest.mark.parametrize("offset", [0, 3])
def test_ranges(sizes, offset):
    ctx, _, _ = G.env()
    t = [torch.ones(s + 16, device="cuda") for s in sizes]
    torch.cuda.synchronize()
    ctx.zero_ranges(*(v for x, s in zip(t, sizes) for v in (x.data_ptr() + 4 * offset, s)))
    ctx.synchronize()
    for x, s in zip(t, sizes):
        assert float(x[:offset].sum()) == offset and not bool(x[offset:offset + s].any())
        assert bool((x[offset + s:] == 1).all())


def test_step_in_batches_of_few_norms():
    """Batches that the norms do not divide into give the gradients of one batch."""
    from autograd_b200.step import FusedLayerStep, StepConfig
    env = G.env()
    cfg = StepConfig(n_layer=3, n_embd=128, n_head=1, head_dim=128, seq_len=40, vocab=392, batch=3)
    got = []
    for batch in (7, 3, 1):
        st = FusedLayerStep(*env, cfg, seed=9)
        st._batch = batch
        env[0].copy_from_host(st.ids, np.arange(120, dtype=np.int32))
        env[0].copy_from_host(st.targets, np.arange(120, dtype=np.int32)[::-1].copy())
        st.forward()
        st.backward()
        got.append(env[0].copy_to_host(st.small_bucket, (st.n_small,), np.uint32).copy())
        st.close()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2]) and got[0].any()
