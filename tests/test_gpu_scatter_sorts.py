"""Scatter-adds on both sides of the sizes where the sort, its digits per thread, its passes and the groups of sorted entries
change hands.  Small whole numbers: their sums are exact in any order, so every row has to be equal to the last bit."""
import pytest
import torch

import autograd_b200 as ag
import gpu_util as G

pytestmark = pytest.mark.gpu


def _run(n, c, v, bf16, bad, frequent):
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda")
    g.manual_seed(n + c + v)
    ids = torch.randint(0, v, (n,), device="cuda", generator=g, dtype=torch.int32)
    if frequent:
        ids[torch.rand(n, device="cuda", generator=g) < 0.4] = v - 1
    if bad:
        ids[::97], ids[5::101] = v, -3
    dout = torch.randint(-8, 9, (n, c), device="cuda", generator=g).float()
    table = torch.randint(-8, 9, (v, c), device="cuda", generator=g).float()
    ok = (ids >= 0) & (ids < v)
    want = table.double().index_add(0, ids[ok].long(), dout[ok].double())
    if bf16:
        want, table = want.float().bfloat16(), table.bfloat16()
    scratch = torch.empty(ctx.scatter_add_scratch_bytes(n, c, v), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    call = ctx.gather_backward_bf16 if bf16 else ctx.gather_backward
    call(ids.data_ptr(), dout.data_ptr(), table.data_ptr(), scratch.data_ptr(), scratch.numel(), n, c, v)
    ctx.synchronize()
    if bad:
        with pytest.raises(ag.AgError):
            ctx.check_status()
    G.check_clean_status()
    assert torch.equal(table.float() if bf16 else table.double(), want.float() if bf16 else want)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("frequent", [False, True])
@pytest.mark.parametrize("n,c,v", [
    (257, 1283, 1), (1024, 1540, 511), (1025, 4, 512), (2048, 36, 513), (2049, 4, 300), (4096, 5, 262143), (4096, 4, 262144),
    (4097, 4, 262144),                                                          # one CTA, or three passes in launches
    (6144, 406, 3000), (6145, 406, 3000), (12500, 64, 70), (12501, 64, 70),     # groups of 8 or 16
    (6000, 750, 3000), (6001, 750, 3000),                                       # 16 or 32
    (24575, 326, 500), (24576, 326, 500), (24577, 325, 500)])                   # 32 or 64, or too few elements
def test_sizes(n, c, v, frequent, bf16):
    _run(n, c, v, bf16, False, frequent)


@pytest.mark.parametrize("n", [1025, 3000, 4096])
def test_ids_outside_the_table(n):
    _run(n, 8, 600, False, True, True)
