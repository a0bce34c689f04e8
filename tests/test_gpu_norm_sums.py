"""Column sums of norms of many rows against exact ones, a batch of them that is refused, and rows of the wide norms' backward that
are read ahead of what is written: in place, and beside rows with Inf and NaN."""
import ctypes

import pytest
import torch

import gpu_util as G
from autograd_b200 import AgError
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


def _partials(ctx, c, norms=1):
    nbytes = ctx.norm_partials_bytes(c)
    return torch.zeros(norms, nbytes // 4, device="cuda"), nbytes


@pytest.mark.parametrize("n,c", [(4096, 128), (4104, 128), (4104, 132), (9000, 128), (9001, 36)])
def test_sums_of_many_partial_rows(n, c):
    """512 partial rows, one more, and two rounds of loads.  Whole-number dy: dbeta is exact in any order."""
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda").manual_seed(n + c)
    dy = torch.randint(-8, 9, (2, n, c), device="cuda", generator=g).float()
    x, gamma = torch.randn(2, n, c, device="cuda", generator=g), torch.randn(2, c, device="cuda", generator=g)
    dx = torch.empty_like(x)
    one, two = torch.zeros(2, 2, c, device="cuda"), torch.zeros(2, 2, c, device="cuda")
    part, nbytes = _partials(ctx, c, 2)
    rows = (ctypes.c_int32 * 2)()
    torch.cuda.synchronize()
    for i in range(2):
        a = [t[i].data_ptr() for t in (dy, x, gamma)] + [0, dx[i].data_ptr()]
        ctx.layernorm_backward(*a, one[i, 0].data_ptr(), one[i, 1].data_ptr(), part.data_ptr(), nbytes, n, c, 1e-5)
    for i in range(2):
        a = [t[i].data_ptr() for t in (dy, x, gamma)] + [0, dx[i].data_ptr()]
        ctx.layernorm_backward_rows(*a, part[i].data_ptr(), nbytes, ctypes.addressof(rows) + 4 * i, n, c, 1e-5)
    ctx.norm_partials_add(part.data_ptr(), nbytes // 4, ctypes.addressof(rows), 2, c, two.data_ptr())
    ctx.synchronize()
    xd = x.double()
    mean, var = xd.mean(2, keepdim=True), xd.var(2, unbiased=False, keepdim=True)
    terms = dy.double() * (xd - mean) / torch.sqrt(var + 1e-5)
    # a term is off by a few 2^-24 of dy, whose norm is about that of the terms, and a sum by as much per addition
    bound = 8 * 2.0 ** -24 * n ** 0.5 * dy.double().norm(dim=1)
    for got in (one, two):
        assert torch.equal(got[:, 1].double(), dy.double().sum(1))
        assert bool(((got[:, 0].double() - terms.sum(1)).abs() <= bound).all())
    G.check_clean_status()


def test_a_refused_batch_adds_nothing():
    """The row count of the last of 65 norms, which a second launch would take."""
    ctx, _, _ = G.env()
    c, norms = 36, 65
    part, nbytes = _partials(ctx, c, norms)
    part.fill_(1.0)
    out = torch.zeros(norms, 2, c, device="cuda")
    rows = (ctypes.c_int32 * norms)(*([1] * norms))
    torch.cuda.synchronize()
    for bad in (nbytes // (8 * c) + 1, -1):
        rows[64] = bad
        with pytest.raises(AgError):
            ctx.norm_partials_add(part.data_ptr(), nbytes // 4, ctypes.addressof(rows), norms, c, out.data_ptr())
        ctx.synchronize()
        assert not bool(out.any())
    rows[64] = 1
    ctx.norm_partials_add(part.data_ptr(), nbytes // 4, ctypes.addressof(rows), norms, c, out.data_ptr())
    ctx.synchronize()
    assert bool((out == 1).all())


@pytest.mark.parametrize("kind,dtype", [("rms", torch.float32), ("rms", torch.bfloat16), ("layer", torch.float32)])
@pytest.mark.parametrize("n,c", [(2100, 2048), (700, 2560), (1201, 3928), (450, 5120)])
def test_wide_rows(kind, dtype, n, c):
    """dx over the residual gradient gives the bits of dx beside it; a row with Inf or NaN spoils its own dx only."""
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda").manual_seed(c)
    dy, x, res = (torch.randn(n, c, device="cuda", generator=g).to(dtype) for _ in range(3))
    gamma = torch.randn(c, device="cuda", generator=g)
    part, nbytes = _partials(ctx, c)
    spoilt = {3: float("inf"), n // 2: float("nan"), n - 1: float("-inf")}

    def run(x, dres, dx):
        sums = torch.zeros(2, c, device="cuda")
        torch.cuda.synchronize()
        if kind == "rms":
            ctx.rmsnorm_backward(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), dres.data_ptr(), dx.data_ptr(), sums.data_ptr(),
                                 part.data_ptr(), nbytes, n, c, 1e-6, N.AG_BF16 if dtype == torch.bfloat16 else N.AG_F32)
        else:
            ctx.layernorm_backward(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), dres.data_ptr(), dx.data_ptr(),
                                   sums[0].data_ptr(), sums[1].data_ptr(), part.data_ptr(), nbytes, n, c, 1e-6)
        ctx.synchronize()
        return dx.clone(), sums

    apart, sums = run(x, res, torch.empty_like(x))
    inside = res.clone()
    over, sums2 = run(x, inside, inside)
    assert torch.equal(apart, over) and torch.equal(sums, sums2) and bool(torch.isfinite(apart).all())
    bad = x.clone()
    for r, v in spoilt.items():
        bad[r, 7] = v
    got, sums = run(bad, res, torch.empty_like(x))
    others = torch.tensor([r for r in range(n) if r not in spoilt], device="cuda")
    assert torch.equal(got[others], apart[others])
    assert not bool(torch.isfinite(got[list(spoilt), 7]).any())
    assert not bool(torch.isfinite(sums[0, 7]))
    G.check_clean_status()
