"""The fp32-grade head and projection on scaled fp16 operand pairs: sizes at the edges of tiles, chains and panels, and
operands whose rows and columns differ by many powers of two, against float64 (torch) on the same inputs."""
import numpy as np
import pytest

import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


def _head(X, W, Y, chunk=4096):
    ctx, alloc, be = G.env()
    be.ce_precision, be.ce_vocab_chunk, be.ce_reduction, be.ce_ignore_mode = N.AG_CE_3XTF32, chunk, 0, 0
    x, w, y = G.up(X, grad=0), G.up(W, grad=0), G.up(Y, requires_grad=False)
    loss = G.empty((1,), grad=np.ones(1, np.float32))
    n = G.node("FusedLinearCrossEntropyOp", (x, w, y), (loss,))
    G.run_forward(n)
    G.run_backward(n)
    out = float(G.down(loss)[0]), G.down(x.grad), G.down(w.grad)
    be.ce_vocab_chunk = 4096
    G.check_clean_status()
    G.free(x, w, y, loss)
    return out


def _head_f64(X, W, Y):
    X, W = X.astype(np.float64), W.astype(np.float64)
    L = X @ W.T
    m = L.max(axis=1, keepdims=True)
    lse = m[:, 0] + np.log(np.exp(L - m).sum(axis=1))
    live = (Y >= 0) & (Y < W.shape[0])
    rows = np.flatnonzero(live)
    P = np.exp(L - lse[:, None])
    P[rows, Y[rows]] -= 1.0
    P[~live] = 0.0
    P /= len(Y)
    return float((lse[rows] - L[rows, Y[rows]]).sum() / len(Y)), P @ W, P.T @ X


def _worst_row(got, ref):
    """Largest error of a row of `got`, in norms of that row."""
    norm = np.linalg.norm(ref, axis=1)
    keep = norm > 0
    return float((np.linalg.norm(got[keep] - ref[keep], axis=1) / norm[keep]).max())


@pytest.mark.parametrize("n,c,v", [(1, 32, 32), (128, 64, 257), (129, 772, 1000), (256, 768, 4096), (257, 36, 4104),
                                   (385, 1540, 513), (1000, 100, 8193)])
def test_head_at_tile_edges(n, c, v):
    rng = np.random.default_rng(n + c + v)
    X = rng.standard_normal((n, c)).astype(np.float32)
    W = (0.05 * rng.standard_normal((v, c))).astype(np.float32)
    Y = rng.integers(0, v, n).astype(np.int32)
    Y[1:][rng.random(n - 1) < 0.1] = -1
    loss, dX, dW = _head(X, W, Y)
    r_loss, r_dX, r_dW = _head_f64(X, W, Y)
    assert abs(loss - r_loss) <= 1e-5 * max(abs(r_loss), 1e-3)
    live = np.abs(r_dX).sum(axis=1) > 0
    assert not dX[~live].any()
    assert _worst_row(dX, r_dX) < 3e-5 and _worst_row(dW, r_dW) < 1e-4


def test_rows_columns_and_tokens_of_very_different_size():
    """Activations with outlier channels, rows of W that are tiny or zero, and tokens whose probability is far below
    the range of one fp16 scale (down to e^-45): every gradient row keeps its relative accuracy."""
    rng = np.random.default_rng(7)
    n, c, v = 700, 200, 3000
    X = rng.standard_normal((n, c)).astype(np.float32)
    X[:, ::67] *= 100.0
    X[:, 1] = 8.0
    W = (0.02 * rng.standard_normal((v, c))).astype(np.float32)
    W[:, ::67] *= 0.01
    W[v // 2:, 1] = -(5.5 * rng.random(v - v // 2)).astype(np.float32)   # unlikely tokens
    W[5], W[6] = 0.0, W[6] * 1e-9
    Y = rng.integers(0, v // 2, n).astype(np.int32)
    loss, dX, dW = _head(X, W, Y, chunk=1024)
    r_loss, r_dX, r_dW = _head_f64(X, W, Y)
    assert abs(loss - r_loss) <= 1e-5 * abs(r_loss)
    assert _worst_row(dX, r_dX) < 1e-4
    assert _worst_row(dW, r_dW) < 1e-3   # the fp32 logits themselves are worth 1e-5 of e^logit times their size


@pytest.mark.parametrize("n,k,c", [(1, 64, 32), (129, 388, 36), (256, 384, 256), (1000, 1540, 100)])
def test_projection_at_tile_edges(n, k, c):
    ctx, alloc, be = G.env()
    be.ce_precision = N.AG_CE_3XTF32
    rng = np.random.default_rng(n + k + c)
    x_, act_ = rng.standard_normal((n, c), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    act_ *= np.exp(3 * rng.standard_normal((n, 1))).astype(np.float32)
    w_ = (rng.standard_normal((k, c)) * np.exp(2 * rng.standard_normal((1, c)))).astype(np.float32)
    b_, dout_ = rng.standard_normal(c, dtype=np.float32), rng.standard_normal((n, c), dtype=np.float32)
    x, act, w, b = (G.up(a, grad=0) for a in (x_, act_, w_, b_))
    out = G.empty((n, c), grad=dout_)
    node = G.node("FusedLinearAddOp", (x, act, w, b), (out,))
    G.run_forward(node)
    G.run_backward(node)
    A, Wd, D = act_.astype(np.float64), w_.astype(np.float64), dout_.astype(np.float64)
    scale = np.abs(A) @ np.abs(Wd) + np.abs(b_) + np.abs(x_)
    assert (np.abs(G.down(out) - (A @ Wd + b_ + x_)) / scale).max() < 3e-6
    assert (np.abs(G.down(act.grad) - D @ Wd.T) / (np.abs(D) @ np.abs(Wd.T))).max() < 1e-5
    assert (np.abs(G.down(w.grad) - A.T @ D) / (np.abs(A.T) @ np.abs(D))).max() < 1e-5
    G.check_clean_status()
    G.free(x, act, w, b, out)
