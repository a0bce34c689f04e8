"""Heads and projections of few multiply-adds, whose operands are split inside the products: sizes at the edges of tiles, stages
and splits in every precision, against float64 (torch); the same for the operand pairs of larger ones, which the smaller sizes
of the other files no longer reach."""
import numpy as np
import pytest
import torch

import gpu_util as G
import test_gpu_head_operands as H
import test_gpu_operand_ranges as R
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu

# A product errs by 2^-23 (three parts), 2^-16 (two) or 2^-8 (one) of the sizes of its terms, the sums by some 2^-24 per
# addition of a chain of 144: in the 2-norm of a result, whose terms cancel to a tenth of their sizes or so.
BOUND = {N.AG_CE_3XTF32: 5e-6, N.AG_CE_BF16X3: 3e-5, N.AG_CE_BF16: 8e-3}
MODES = list(BOUND)


def _off(got, ref):
    ref = ref.cpu().numpy()
    return float(np.linalg.norm(got - ref) / max(np.linalg.norm(ref), 1e-300))


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


@pytest.mark.parametrize("precision", MODES)
@pytest.mark.parametrize("weighted,reduction,dloss", [(False, 0, 1.0), (False, 1, 3e-7), (True, 0, 2.0 ** 40)])
@pytest.mark.parametrize("n,c,v", [(1, 32, 32), (128, 64, 129), (127, 120, 64), (129, 72, 4608), (64, 2304, 200), (4097, 40, 2305),
                                   (2305, 64, 300), (257, 136, 5003)])
def test_head(n, c, v, weighted, reduction, dloss, precision):
    ctx, alloc, be = G.env()
    be.ce_precision, be.ce_vocab_chunk, be.ce_reduction, be.ce_ignore_mode = precision, 4096, reduction, 0
    rng = np.random.default_rng(n + c + v)
    X, W = rng.standard_normal((n, c), dtype=np.float32), (0.05 * rng.standard_normal((v, c))).astype(np.float32)
    Y = rng.integers(0, v, n).astype(np.int32)
    Y[1:][rng.random(n - 1) < 0.1] = -1
    weight = (rng.random(n) / n).astype(np.float32)
    x, w, y = G.up(X, grad=0), G.up(W, grad=0), G.up(Y, requires_grad=False)
    extra = (G.up(weight, requires_grad=False),) if weighted else ()
    loss = G.empty((1,), grad=np.full(1, dloss, np.float32))
    node = G.node("FusedLinearCrossEntropyOp", (x, w, y) + extra, (loss,))
    G.run_forward(node)
    G.run_backward(node)
    got = float(G.down(loss)[0]), G.down(x.grad), G.down(w.grad)
    G.run_backward(node)  # once more: added to what is there (split contractions add their parts one by one)
    for grad, first in ((x.grad, got[1]), (w.grad, got[2])):
        assert np.linalg.norm(G.down(grad) - 2 * first) <= 1e-6 * np.linalg.norm(first)
        be.fill_storage2(grad.storage, 0)
    G.run_backward(node)  # and from zero: the same bits
    assert np.array_equal(G.down(x.grad), got[1]) and np.array_equal(G.down(w.grad), got[2])
    Xd, Wd, t = _f64(X), _f64(W), torch.from_numpy(Y).cuda().long()
    if precision == N.AG_CE_BF16:  # the logits are those of the rounded operands
        Xd, Wd = (a.float().bfloat16().double() for a in (Xd, Wd))
    L = Xd @ Wd.T
    lse = torch.logsumexp(L, 1)
    live = t >= 0
    each = torch.where(live, lse - L.gather(1, t.clamp(min=0)[:, None])[:, 0], 0.0)
    scale = _f64(weight) if weighted else torch.full((n,), 1.0 / (n if reduction == 0 else int(live.sum())), device="cuda").double()
    p = torch.exp(L - lse[:, None])
    p[live.nonzero()[:, 0], t[live]] -= 1.0
    p *= (scale * live * dloss)[:, None]
    assert abs(got[0] - float((each * scale).sum())) <= (1e-4 if precision == N.AG_CE_BF16 else 2e-6) * float((each * scale).sum())
    assert _off(got[1], p @ Wd) < BOUND[precision] and _off(got[2], p.T @ Xd) < BOUND[precision]
    assert not got[1][~live.cpu().numpy()].any()
    G.check_clean_status()
    G.free(x, w, y, loss, *extra)


@pytest.mark.parametrize("precision", [N.AG_CE_3XTF32, N.AG_CE_BF16])
@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("n,k,c", [(1, 8, 8), (128, 128, 128), (129, 1160, 136), (16, 5120, 64), (2049, 72, 136), (300, 64, 2312),
                                   (4700, 64, 40), (16384, 320, 264), (400, 5120, 904)])
def test_projection(n, k, c, offset, precision):
    """`offset` bytes: the products' results and the bias gradient may lie at any word."""
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(n + k + c)
    x, act, dout = (rng.standard_normal(s, dtype=np.float32) for s in ((n, c), (n, k), (n, c)))
    w, b = (0.1 * rng.standard_normal((k, c))).astype(np.float32), rng.standard_normal(c, dtype=np.float32)
    buf = {name: torch.zeros(int(np.prod(s)) + 4, device="cuda") for name, s in
           (("out", (n, c)), ("dx", (n, c)), ("dact", (n, k)), ("dw", (k, c)), ("db", (c,)))}
    at = {name: t.data_ptr() + (offset if name != "dx" else 0) for name, t in buf.items()}
    inp = {name: torch.from_numpy(a).cuda() for name, a in (("x", x), ("act", act), ("w", w), ("b", b), ("dout", dout))}
    p = {name: t.data_ptr() for name, t in inp.items()}
    nbytes = ctx.linear_add_scratch_bytes(n, k, c, precision)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.linear_add_forward(p["x"], p["act"], p["w"], p["b"], at["out"], n, k, c, precision, scratch.data_ptr(), nbytes)
    ctx.linear_add_backward(p["dout"], p["act"], p["w"], at["dx"], at["dact"], at["dw"], at["db"], n, k, c, precision,
                            scratch.data_ptr(), nbytes)
    ctx.synchronize()
    X, A, D, Wd = (_f64(a) for a in (x, act, dout, w))
    if precision == N.AG_CE_BF16:
        A, Wd = (a.float().bfloat16().double() for a in (A, Wd))
    Db = D.float().bfloat16().double() if precision == N.AG_CE_BF16 else D
    bound = 1e-6 if precision == N.AG_CE_BF16 else BOUND[precision]  # the rounded operands are the oracle's too
    for name, ref in (("out", A @ Wd + _f64(b) + X), ("dx", D), ("dact", Db @ Wd.T), ("dw", A.T @ Db), ("db", D.sum(0))):
        first = (at[name] - buf[name].data_ptr()) // 4
        got = buf[name][first:first + ref.numel()].view(ref.shape).cpu().numpy()
        assert _off(got, ref) < max(bound, 1e-6), name
    G.check_clean_status()


def test_short_scratch_and_a_residual_gradient_off_its_packets_are_refused():
    ctx, _, _ = G.env()
    d = ctx.flce_desc(40, 64, 300, precision=N.AG_CE_3XTF32)
    mem = G.empty((1 << 16,))
    a = mem.storage.ptr.address
    with pytest.raises(N.AgError, match="scratch"):
        ctx.flce_forward(d, a, a, a, 0, a, a, a, ctx.flce_scratch_bytes(d) - 1)
    with pytest.raises(N.AgError, match="scratch"):
        ctx.linear_add_forward(a, a, a, a, a, 8, 64, 64, N.AG_CE_3XTF32, a, ctx.linear_add_scratch_bytes(8, 64, 64, 1) - 1)
    with pytest.raises(N.AgError, match="aligned"):
        ctx.linear_add_backward(a, a, a, a + 4, a, a, a, 8, 64, 64, N.AG_CE_3XTF32, a, 1 << 18)
    G.free(mem)


# ---------------------------------------------------------------------------- operand pairs, at sizes that still take them
@pytest.mark.parametrize("n,c,v", [(1200, 516, 4104), (2560, 772, 1153)])
def test_pair_head_at_tile_edges(n, c, v):
    H.test_head_at_tile_edges(n, c, v)


@pytest.mark.parametrize("n,k,c", [(2300, 1028, 1060), (8192, 516, 644)])
def test_pair_projection_at_tile_edges(n, k, c):
    H.test_projection_at_tile_edges(n, k, c)


@pytest.mark.parametrize("index", ["inner", "columns", "rows"])
@pytest.mark.parametrize("power", [0, 27, 100, None])
@pytest.mark.parametrize("n,k,c", [(2300, 1028, 1060), (1100, 1540, 1636)])
def test_pair_projection_ranges(n, k, c, power, index):
    R.test_projection(n, k, c, power, index)


@pytest.mark.parametrize("power", [0, 27, 100, None])
def test_pair_head_with_outlier_channels(power):
    R.test_head_with_outlier_channels(1400, 520, 3400, power)


@pytest.mark.parametrize("power", [0, 24, 30])
def test_pair_head_with_a_large_row_of_an_unlikely_token(power):
    R.test_head_with_a_large_row_of_an_unlikely_token(1400, 520, 3400, power)


@pytest.mark.parametrize("power", [0, 30])
def test_pair_zero_tiny_and_nonfinite_elements(power):
    R.test_zero_tiny_and_nonfinite_elements(1100, 1540, 1636, power)


@pytest.mark.parametrize("dloss", [1.0, 2.0 ** -60, 2.0 ** 40, 2.0 ** 60])
def test_probabilities_keep_their_bits_at_any_loss_gradient(dloss):
    """W holds the logits beside a unit matrix, so that dX shows the gradients of the logits themselves.  A logit below 4 in size
    less the row's logarithm is rounded by 1.2e-7, the exponent of 2 (below 6) by 2.4e-7 ln 2, the exponential by 2^-22, the
    logarithm by 1.2e-7: 6.5e-7 of p in all.  (With the scale of the loss gradient in the exponent of p it is 3e-6 at 2^-60.)"""
    ctx, alloc, be = G.env()
    be.ce_precision, be.ce_vocab_chunk, be.ce_reduction, be.ce_ignore_mode = N.AG_CE_3XTF32, 4096, 0, 0
    rng = np.random.default_rng(3)
    n = v = 40
    W = np.zeros((v, v + 4), np.float32)
    W[:, 0] = np.round(np.log(rng.dirichlet(np.full(v, 100.0))) * 4096) / 4096  # exact in the products too
    W[:, 4:] = np.eye(v, dtype=np.float32)
    X = np.zeros((n, v + 4), np.float32)
    X[:, 0] = 1.0
    Y = rng.integers(0, v, n).astype(np.int32)
    x, w, y = G.up(X, grad=0), G.up(W, grad=0), G.up(Y, requires_grad=False)
    loss = G.empty((1,), grad=np.full(1, dloss, np.float32))
    node = G.node("FusedLinearCrossEntropyOp", (x, w, y), (loss,))
    G.run_forward(node)
    G.run_backward(node)
    got = G.down(x.grad)[:, 4:].astype(np.float64) * n / dloss
    L = X[:, :1].astype(np.float64) * W[:, 0].astype(np.float64)[None, :]
    P = np.exp(L - L.max(1, keepdims=True))
    P /= P.sum(1, keepdims=True)
    P[np.arange(n), Y] -= 1.0
    err = float((np.abs(got - P) / np.abs(P)).max())
    print("loss gradient %g: %.1e" % (dloss, err))
    assert err < 8e-7
    G.check_clean_status()
    G.free(x, w, y, loss)


@pytest.mark.parametrize("power", [-100, -108, -114, -120, -124])
def test_operands_at_the_lower_end_of_the_exponents(power):
    """The parts of an operand are bf16 words, which end at 2^-133.  Elements above 2^-110 keep their 24 bits; smaller ones are off
    by 2^-134 at most, doubled here for the products that are left out."""
    ctx, alloc, be = G.env()
    be.ce_precision = N.AG_CE_3XTF32
    rng = np.random.default_rng(5)
    n, k, c = 100, 96, 64
    act_ = np.ldexp(rng.standard_normal((n, k)), power).astype(np.float32)
    w_, dout_ = (rng.standard_normal(s, dtype=np.float32) for s in ((k, c), (n, c)))
    act, w = G.up(act_, grad=0), G.up(w_, grad=0)
    x, b = G.up(np.zeros((n, c), np.float32), grad=0), G.up(np.zeros(c, np.float32), grad=0)
    out = G.empty((n, c), grad=dout_)
    node = G.node("FusedLinearAddOp", (x, act, w, b), (out,))
    G.run_forward(node)
    G.run_backward(node)
    for name, got, p, q in (("out", G.down(out), act_, w_), ("dw", G.down(w.grad), act_.T, dout_)):
        p, q = p.astype(np.float64), q.astype(np.float64)
        size, other = np.abs(p) @ np.abs(q), np.ones_like(p) @ np.abs(q)
        err = np.abs(got - p @ q)
        print(name, "2^%d: %.1e of the terms, 2^-133 x %.2f" % (power, (err / size).max(), (err / (2.0 ** -133 * other)).max()))
        assert (err <= 3e-6 * size + 2.0 ** -133 * other).all(), name
    G.check_clean_status()
    G.free(x, act, w, b, out)


@pytest.mark.parametrize("precision", [N.AG_CE_3XTF32, N.AG_CE_BF16])
@pytest.mark.parametrize("n,k,c", [(1023, 64, 72), (1024, 64, 72), (1535, 72, 1544), (1536, 64, 1536)])
def test_projection_where_the_bias_gradient_changes_hands(n, k, c, precision):
    test_projection(n, k, c, 0, precision)


@pytest.mark.parametrize("n", [32768, 32769])
def test_head_where_counting_the_rows_changes_hands(n):
    test_head(n, 32, 64, False, 1, 1.0, N.AG_CE_3XTF32)
