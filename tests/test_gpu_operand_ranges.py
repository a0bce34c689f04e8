"""fp32-grade products whose operands differ by many powers of two along the contraction index: where an element of one
operand is large, the elements of the other that it meets are small, so that every product counts.  One element of the
index far from the others (as an outlier channel whose weights are small), and all of them spread.  Errors against
float64, relative to the sum of the products' sizes."""
import numpy as np
import pytest

import gpu_util as G
from autograd_b200 import _native as N
from conftest import assert_close

pytestmark = pytest.mark.gpu

POWERS = [0, 8, 10, 20, 24, 27, 30, 60, 100]


def _exponents(n, power, seed):
    """Index 3 by 2^power, the others by 1; or all of them spread over +-40 powers of two."""
    if power is None:
        return np.random.default_rng(seed).integers(-40, 41, n)
    e = np.zeros(n, np.int64)
    e[3] = power
    return e


def _rel(got, a, b, extra=0.0):
    """Largest error of a . b + extra over the sum of the sizes of its terms."""
    a, b, extra = a.astype(np.float64), b.astype(np.float64), np.asarray(extra, np.float64)
    return float((np.abs(got - (a @ b + extra)) / (np.abs(a) @ np.abs(b) + np.abs(extra))).max())


def _scaled(rng, shape, axis, e):
    x = rng.standard_normal(shape, dtype=np.float32)
    return np.ldexp(x, e[:, None] if axis == 0 else e[None, :]).astype(np.float32)


@pytest.mark.parametrize("index", ["inner", "columns", "rows"])
@pytest.mark.parametrize("power", POWERS + [None])
@pytest.mark.parametrize("n,k,c", [(300, 520, 132), (600, 256, 64), (40, 128, 32), (128, 132, 36), (129, 128, 36), (2048, 64, 32),
                                   (2049, 64, 40)])
def test_projection(n, k, c, power, index):
    """`index`: the one that the forward, the activation gradient or the weight gradient contracts."""
    ctx, alloc, be = G.env()
    be.ce_precision = N.AG_CE_3XTF32
    rng = np.random.default_rng(n + k + c)
    e = {"inner": np.zeros(k, np.int64), "columns": np.zeros(c, np.int64), "rows": np.zeros(n, np.int64)}
    e[index] = _exponents(len(e[index]), power, k)
    act_, w_, dout_ = (rng.standard_normal(s, dtype=np.float32) for s in ((n, k), (k, c), (n, c)))
    act_ = np.ldexp(np.ldexp(act_, e["inner"][None, :]), e["rows"][:, None]).astype(np.float32)
    w_ = np.ldexp(np.ldexp(w_, -e["inner"][:, None]), -e["columns"][None, :]).astype(np.float32)
    dout_ = np.ldexp(np.ldexp(dout_, e["columns"][None, :]), -e["rows"][:, None]).astype(np.float32)
    act, w = G.up(act_, grad=0), G.up(w_, grad=0)
    x, b = G.up(np.zeros((n, c), np.float32), grad=0), G.up(np.zeros(c, np.float32), grad=0)
    out = G.empty((n, c), grad=dout_)
    node = G.node("FusedLinearAddOp", (x, act, w, b), (out,))
    G.run_forward(node)
    G.run_backward(node)
    errs = _rel(G.down(out), act_, w_), _rel(G.down(act.grad), dout_, w_.T), _rel(G.down(w.grad), act_.T, dout_)
    print(f"{index} 2^{power}: " + " ".join("%.1e" % v for v in errs))
    assert errs[0] < 3e-6 and errs[1] < 1e-5 and errs[2] < 1e-5
    G.check_clean_status()
    G.free(x, act, w, b, out)


def _head(X, W, Y):
    ctx, alloc, be = G.env()
    be.ce_precision, be.ce_vocab_chunk, be.ce_reduction, be.ce_ignore_mode = N.AG_CE_3XTF32, 4096, 0, 0
    x, w, y = G.up(X, grad=0), G.up(W, grad=0), G.up(Y, requires_grad=False)
    loss = G.empty((1,), grad=np.ones(1, np.float32))
    node = G.node("FusedLinearCrossEntropyOp", (x, w, y), (loss,))
    G.run_forward(node)
    G.run_backward(node)
    out = float(G.down(loss)[0]), G.down(x.grad).astype(np.float64), G.down(w.grad).astype(np.float64)
    G.check_clean_status()
    G.free(x, w, y, loss)
    return out


def _head_f64(X, W, Y):
    X, W = X.astype(np.float64), W.astype(np.float64)
    L = X @ W.T
    m = L.max(axis=1, keepdims=True)
    lse = m[:, 0] + np.log(np.exp(L - m).sum(axis=1))
    rows = np.arange(len(Y))
    P = np.exp(L - lse[:, None])
    P[rows, Y] -= 1.0
    P /= len(Y)
    return float((lse - L[rows, Y]).mean()), P @ W, P.T @ X


@pytest.mark.parametrize("power", POWERS + [None])
@pytest.mark.parametrize("n,c,v", [(300, 132, 1000), (700, 64, 300)])
def test_head_with_outlier_channels(n, c, v, power):
    rng = np.random.default_rng(n + c + v)
    e = _exponents(c, power, c)
    X, W = _scaled(rng, (n, c), 1, e), _scaled(rng, (v, c), 1, -e) * np.float32(0.1)
    Y = rng.integers(0, v, n).astype(np.int32)
    loss, dX, dW = _head(X, W, Y)
    r_loss, r_dX, r_dW = _head_f64(X, W, Y)
    assert abs(loss - r_loss) <= 1e-5 * abs(r_loss)
    back = np.ldexp(1.0, e)[None, :]   # dX is as small in a channel as W is, dW as large as X
    assert_close(dX * back, r_dX * back, 3e-5, "dX")
    assert_close(dW / back, r_dW / back, 1e-4, "dW")


@pytest.mark.parametrize("power", [0, 10, 20, 24, 27, 30])
@pytest.mark.parametrize("n,c,v", [(300, 132, 1000), (600, 64, 300)])
def test_head_with_a_large_row_of_an_unlikely_token(n, c, v, power):
    """A token whose row of W is 2^power times the others' and whose logit is far below them: nothing of it reaches dX."""
    rng = np.random.default_rng(n + c + v)
    X, W = rng.standard_normal((n, c)).astype(np.float32), (0.1 * rng.standard_normal((v, c))).astype(np.float32)
    X[:, 1] = 4.0
    W[5] = (0.01 * rng.standard_normal(c)).astype(np.float32)
    W[5, 1] = -4.0
    W[5] *= np.float32(2.0 ** power)
    Y = rng.integers(6, v, n).astype(np.int32)
    loss, dX, dW = _head(X, W, Y)
    r_loss, r_dX, r_dW = _head_f64(X, W, Y)
    assert abs(loss - r_loss) <= 1e-5 * abs(r_loss)
    assert_close(dX, r_dX, 3e-5, "dX")
    assert_close(dW, r_dW, 1e-4, "dW")


def test_head_rows_have_to_be_aligned():
    """X is read in 16-byte packets before anything else of the backward: refused by the host."""
    ctx, _, _ = G.env()
    d = ctx.flce_desc(8, 64, 64, precision=N.AG_CE_3XTF32)
    nbytes = ctx.flce_scratch_bytes(d)
    mem = G.empty((nbytes // 4 + 64,))
    a = mem.storage.ptr.address
    with pytest.raises(N.AgError, match="aligned"):
        ctx.flce_backward(d, a + 4, a, a, 0, a, a, a, a, a, nbytes)
    G.free(mem)


@pytest.mark.parametrize("power", [0, 30])
@pytest.mark.parametrize("n,k,c", [(100, 96, 32), (300, 520, 132)])
def test_zero_tiny_and_nonfinite_elements(n, k, c, power):
    """Channels and rows that are zero or far below the others, balanced or not; an Inf or NaN reaches the outputs that it
    belongs to and no others."""
    ctx, alloc, be = G.env()
    be.ce_precision = N.AG_CE_3XTF32
    rng = np.random.default_rng(k)
    act_, w_, dout_ = (rng.standard_normal(s, dtype=np.float32) for s in ((n, k), (k, c), (n, c)))
    act_[:, 3] *= np.float32(2.0 ** power)
    w_[3] *= np.float32(2.0 ** -power)
    act_[:, 5], w_[6], w_[:, 7], dout_[8], act_[9] = 0, 0, 0, 0, 0
    act_[:, 10] *= np.float32(1e-30)
    act_[11, 12], act_[13, 14], w_[15, 16] = np.inf, np.nan, np.inf
    act, w = G.up(act_, grad=0), G.up(w_, grad=0)
    x, b = G.up(np.zeros((n, c), np.float32), grad=0), G.up(np.zeros(c, np.float32), grad=0)
    out = G.empty((n, c), grad=dout_)
    node = G.node("FusedLinearAddOp", (x, act, w, b), (out,))
    G.run_forward(node)
    G.run_backward(node)
    A, W, D = act_.astype(np.float64), w_.astype(np.float64), dout_.astype(np.float64)
    with np.errstate(invalid="ignore"):
        for got, p, q, bound in ((G.down(out), A, W, 3e-6), (G.down(act.grad), D, W.T, 1e-5), (G.down(w.grad), A.T, D, 1e-5)):
            want, size = p @ q, np.abs(p) @ np.abs(q)
            bad = ~np.isfinite(size)
            assert np.array_equal(~np.isfinite(got), bad)
            assert (np.abs(got - want)[~bad] <= bound * size[~bad]).all()
    G.check_clean_status()
    G.free(x, act, w, b, out)
