"""Heads whose logits stay in memory between forward and backward: against float64, beside the head that recomputes them,
at row and column counts that no tile divides, over several panels, with ignored rows, row weights and one gradient only."""
import pytest
import torch

import gpu_util as G
from autograd_b200 import AgError
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


def _inputs(n, c, v, ignored, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(n, c, device="cuda", generator=g)
    w = torch.randn(v, c, device="cuda", generator=g) * 0.05
    t = torch.randint(0, v, (n,), device="cuda", generator=g, dtype=torch.int32)
    if ignored:
        t[::7] = -1
        t[3::11] = v
    return x, w, t, torch.rand(n, device="cuda", generator=g)


def _run(ctx, d, x, w, t, weights, dloss, want_dx, want_dw, keep):
    n, c, v = d.N, d.C, d.V
    lse, loss = torch.zeros(n, device="cuda"), torch.zeros(1, device="cuda")
    dx, dw = torch.full((n, c), 0.5, device="cuda"), torch.full((v, c), -0.25, device="cuda")
    scratch = torch.empty(ctx.flce_scratch_bytes(d), dtype=torch.uint8, device="cuda")
    up = torch.tensor([dloss], device="cuda")
    a = (d, x.data_ptr(), w.data_ptr(), t.data_ptr(), weights.data_ptr() if weights is not None else 0)
    g = (dx.data_ptr() if want_dx else 0, dw.data_ptr() if want_dw else 0)
    s = (scratch.data_ptr(), scratch.numel())
    torch.cuda.synchronize()
    if keep:
        nbytes = ctx.flce_logits_bytes(d)
        kept = torch.full((nbytes // 4,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        ctx.flce_forward_keep(*a, loss.data_ptr(), lse.data_ptr(), kept.data_ptr(), nbytes, *s)
        ctx.synchronize()
        scratch.fill_(0xff)       # nothing but the logits and lse has to outlive the forward call
        torch.cuda.synchronize()
        ctx.flce_backward_kept(*a, up.data_ptr(), lse.data_ptr(), kept.data_ptr(), nbytes, *g, *s)
    else:
        ctx.flce_forward(*a, loss.data_ptr(), lse.data_ptr(), *s)
        ctx.flce_backward(*a, up.data_ptr(), lse.data_ptr(), *g, *s)
    ctx.synchronize()
    G.check_clean_status()
    return float(loss), dx, dw


def _exact(d, x, w, t, weights, dloss):
    n, v = d.N, d.V
    x, w = x.double(), w.double()
    if d.precision == N.AG_CE_BF16:
        x, w = x.float().bfloat16().double(), w.float().bfloat16().double()
    z = x @ w.T
    lse = torch.logsumexp(z, 1)
    ok = (t >= 0) & (t < v)
    at = t.long().clamp(0, v - 1)
    rows = torch.where(ok, lse - z.gather(1, at[:, None])[:, 0], 0.0)
    sc = weights.double() if weights is not None else torch.full_like(
        lse, 1.0 / (n if d.reduction == N.AG_CE_MEAN_ALL_ROWS else max(int(ok.sum()), 1)))
    dl = torch.exp(z - lse[:, None])
    dl[torch.arange(n, device="cuda")[ok], at[ok]] -= 1.0
    dl *= dloss * sc[:, None]
    if d.ignore_mode == N.AG_CE_IGNORE_MASKED:
        dl[~ok] = 0.0
    return float((rows * sc).sum()), dl @ w + 0.5, dl.T @ x - 0.25


def _off(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("n,c,v,chunk,precision,weighted,reduction,ignore,dx,dw", [
    (2001, 392, 5003, 4096, 1, False, 0, 0, True, True),
    (333, 1536, 8200, 4096, 1, True, 0, 0, True, True),       # one panel, wider than vocab_chunk
    (19200, 256, 4100, 1000, 1, False, 1, 0, True, True),     # two row tiles, panels of 1000, 1000, 1000, 1000, 100
    (2500, 1540, 777, 4096, 1, False, 0, 1, True, True),      # rows without a target keep their probabilities
    (2001, 392, 5003, 4096, 1, False, 0, 0, True, False),
    (2001, 392, 5003, 4096, 1, False, 0, 0, False, True),
    (2001, 392, 5003, 4096, 3, False, 1, 0, True, True),
    (19200, 512, 4100, 1000, 3, True, 0, 0, True, True),
    (2001, 392, 5003, 4096, 2, False, 0, 0, True, True),
    (130, 2048, 300007, 4096, 2, True, 0, 0, True, True),
    # products straight from fp32 operands: tiles and packets that no size divides, every mode, reduction and kind of row
    (333, 392, 5003, 4096, 1, False, 1, 0, True, True),
    (128, 64, 1001, 4096, 1, True, 0, 0, True, True),
    (129, 68, 1007, 4096, 1, False, 0, 1, True, True),
    (1, 32, 33, 4096, 1, False, 0, 1, True, True),
    (192, 128, 640, 4096, 3, False, 1, 0, True, False),
    (40, 1536, 20000, 4096, 2, False, 0, 0, True, True),
    (33000, 64, 66, 4096, 1, False, 1, 0, False, True),
])
def test_kept_logits(n, c, v, chunk, precision, weighted, reduction, ignore, dx, dw):
    ctx, _, _ = G.env()
    d = ctx.flce_desc(n, c, v, vocab_chunk=chunk, precision=precision, reduction=reduction, ignore_mode=ignore)
    assert ctx.flce_logits_bytes(d) == 4 * n * ((v + 31) // 32 * 32)
    x, w, t, weights = _inputs(n, c, v, True, n + v)
    weights = weights if weighted else None
    want = _exact(d, x, w, t, weights, 0.5)
    kept = _run(ctx, d, x, w, t, weights, 0.5, dx, dw, True)
    again = _run(ctx, d, x, w, t, weights, 0.5, dx, dw, False)
    # what tests of the recomputing head allow; and no further from float64 than it, but for its rounding (2^-20)
    tol = 2e-2 if precision == N.AG_CE_BF16 else 1e-4
    assert abs(kept[0] - want[0]) <= 1e-5 * abs(want[0]) and kept[0] == again[0]
    for i, have in ((1, dx), (2, dw)):
        if have:
            off = _off(kept[i], want[i]), _off(again[i], want[i])
            print(f"{'dX' if i == 1 else 'dW'}: {off[0]:.2e}, recomputed {off[1]:.2e}")
            assert off[0] <= tol and off[0] <= 1.02 * off[1] + 2.0 ** -20
        else:
            assert bool((kept[i] == (0.5 if i == 1 else -0.25)).all())


def test_columns_that_no_row_predicts():
    """The gradient of a token whose probability is 1e-12 everywhere, against its own size."""
    ctx, _, _ = G.env()
    n, c, v = 2048, 256, 8192
    d = ctx.flce_desc(n, c, v, precision=N.AG_CE_3XTF32)
    x, w, t, _ = _inputs(n, c, v, False, 5)
    x[:, 0] = 20.0
    w[100:200, 0] = -1.4
    t[(t >= 100) & (t < 200)] = 7
    dw = torch.zeros_like(w)
    scratch = torch.empty(ctx.flce_scratch_bytes(d), dtype=torch.uint8, device="cuda")
    nbytes = ctx.flce_logits_bytes(d)
    logits, lse, loss = torch.empty(nbytes // 4, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(1, device="cuda")
    one = torch.ones(1, device="cuda")
    a, s = (d, x.data_ptr(), w.data_ptr(), t.data_ptr(), 0), (scratch.data_ptr(), scratch.numel())
    torch.cuda.synchronize()
    ctx.flce_forward_keep(*a, loss.data_ptr(), lse.data_ptr(), logits.data_ptr(), nbytes, *s)
    ctx.flce_backward_kept(*a, one.data_ptr(), lse.data_ptr(), logits.data_ptr(), nbytes, 0, dw.data_ptr(), *s)
    ctx.synchronize()
    z = x.double() @ w.double().T
    p = torch.exp(z - torch.logsumexp(z, 1)[:, None])[:, 100:200] / n
    want = p.T @ x.double()
    worst = float(((dw[100:200].double() - want).norm(dim=1) / want.norm(dim=1)).max())
    print(f"dW of columns of {float(p.max()) * n:.1e}: {worst:.2e} of their size")
    assert worst < 1e-4


def test_refused():
    ctx, _, _ = G.env()
    a = torch.zeros(64, device="cuda")
    p = a.data_ptr()
    exact = ctx.flce_desc(4096, 392, 5003, precision=N.AG_CE_FP32)
    narrow = ctx.flce_desc(4096, 128, 16384, precision=N.AG_CE_3XTF32)
    assert ctx.flce_logits_bytes(exact) == ctx.flce_logits_bytes(narrow) == 0
    d = ctx.flce_desc(2001, 392, 5003, precision=N.AG_CE_3XTF32)
    need = ctx.flce_logits_bytes(d)
    for desc, at, nbytes in ((exact, p, need), (d, p, need - 1), (d, 0, need), (d, p + 4, need)):
        with pytest.raises(AgError):
            ctx.flce_forward_keep(desc, p, p, p, 0, p, p, at, nbytes, p, 1 << 40)
        with pytest.raises(AgError):
            ctx.flce_backward_kept(desc, p, p, p, 0, p, p, at, nbytes, p, p, p, 1 << 40)
