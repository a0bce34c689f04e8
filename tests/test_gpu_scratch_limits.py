"""Scatter-adds and projections whose usual route needs more scratch than another one that serves them too: with exactly the bytes
that a refused call names they take the other, with the bytes of the size functions the usual one."""
import re

import pytest
import torch

import autograd_b200 as ag
import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


def _least(call):
    with pytest.raises(ag.AgError) as e:
        call(1)
    return int(re.search(r"needs (\d+)", str(e.value)).group(1))


@pytest.mark.parametrize("n,c", [(4097, 64), (12500, 64), (16000, 200), (50000, 64)])
def test_scatter(n, c):
    ctx, _, _ = G.env()
    v = 300
    g = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(0, v, (n,), device="cuda", generator=g, dtype=torch.int32)
    dout = torch.randint(-8, 9, (n, c), device="cuda", generator=g).float()
    table = torch.zeros((v, c), device="cuda")
    full = ctx.scatter_add_scratch_bytes(n, c, v)
    scratch = torch.empty(full, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()

    def call(nbytes):
        ctx.gather_backward(ids.data_ptr(), dout.data_ptr(), table.data_ptr(), scratch.data_ptr(), nbytes, n, c, v)

    least = _least(call)
    assert least < full
    want = torch.zeros((v, c), device="cuda", dtype=torch.float64).index_add(0, ids.long(), dout.double())
    for k, nbytes in enumerate((least, full)):  # whole numbers: exact
        call(nbytes)
        ctx.synchronize()
        assert torch.equal(table.double(), (k + 1) * want)
    G.check_clean_status()


@pytest.mark.parametrize("n,k,c", [(2381, 556, 1608), (9344, 380, 636), (16384, 1024, 128)])
def test_projection(n, k, c):
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda").manual_seed(n)
    x, act, dout = (torch.randn(s, device="cuda", generator=g) for s in ((n, c), (n, k), (n, c)))
    w, b = 0.1 * torch.randn((k, c), device="cuda", generator=g), torch.randn(c, device="cuda", generator=g)
    full = ctx.linear_add_scratch_bytes(n, k, c, N.AG_CE_3XTF32)
    scratch = torch.empty(full, dtype=torch.uint8, device="cuda")
    out, dx, dact, dw, db = (torch.zeros(s, device="cuda") for s in ((n, c), (n, c), (n, k), (k, c), (c,)))
    torch.cuda.synchronize()

    def forward(nbytes):
        ctx.linear_add_forward(x.data_ptr(), act.data_ptr(), w.data_ptr(), b.data_ptr(), out.data_ptr(), n, k, c, N.AG_CE_3XTF32,
                               scratch.data_ptr(), nbytes)

    def backward(nbytes):
        ctx.linear_add_backward(dout.data_ptr(), act.data_ptr(), w.data_ptr(), dx.data_ptr(), dact.data_ptr(), dw.data_ptr(),
                                db.data_ptr(), n, k, c, N.AG_CE_3XTF32, scratch.data_ptr(), nbytes)

    D = dout.double()
    refs = {"out": (out, act.double() @ w.double() + b.double() + x.double()), "dact": (dact, D @ w.double().T),
            "dw": (dw, act.double().T @ D), "db": (db, D.sum(0)), "dx": (dx, D)}
    for fwd, bwd in ((_least(forward), _least(backward)), (full, full)):
        assert fwd <= full and bwd <= full
        for t in (dx, dact, dw, db):
            t.zero_()
        torch.cuda.synchronize()
        forward(fwd)
        backward(bwd)
        ctx.synchronize()
        for name, (got, ref) in refs.items():  # the operand pairs' bound, which is the wider one
            assert float((got.double() - ref).norm() / ref.norm()) < 5e-6, name
    G.check_clean_status()
