"""Norms of fp32 rows that no 16-byte packet divides, against float64.  Row lengths at the edges of what a thread and a team hold,
every shift of a row against its packets, one row per team and several, operands that are not aligned, residual gradients in
place, and a workspace that holds fewer partial rows than rows of four teams."""
import numpy as np
import pytest
import torch

import gpu_util as G

pytestmark = pytest.mark.gpu

SHAPES = [(700, 257), (5000, 258), (4000, 319), (4001, 387), (3000, 511), (900, 513), (1777, 1026), (901, 1538), (890, 2049), (1000, 767), (3001, 1023), (900, 4098), (889, 4350), (2000, 514), (900, 8190), (880, 8193), (77, 1025)]


def _f64(t):
    return t.double()


@pytest.mark.parametrize("kind", ["layer", "rms"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,c", SHAPES)
def test_norms(n, c, offset, kind):
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda")
    g.manual_seed(n + c)
    new = lambda *s: torch.randn(int(np.prod(s)) + 8, device="cuda", generator=g)[offset:offset + int(np.prod(s))].view(s)
    x, r, dy, dres, gamma, beta = new(n, c), new(n, c), new(n, c), new(n, c), new(c), new(c)
    pad = torch.full((n * c + 16,), 7.0, device="cuda")
    h, y, dx = (pad.clone()[offset:] for _ in range(3))
    dx[:n * c] = dres.reshape(-1)
    dgamma, dbeta = torch.ones(c, device="cuda"), torch.ones(c, device="cuda")
    nbytes = ctx.norm_partials_bytes(c)
    part = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    eps = 1e-5
    if kind == "layer":
        ctx.add_layernorm_forward(x.data_ptr(), r.data_ptr(), gamma.data_ptr(), beta.data_ptr(), h.data_ptr(), y.data_ptr(), 0, 0, n, c, eps)
        ctx.layernorm_backward(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), dx.data_ptr(), dx.data_ptr(), dgamma.data_ptr(),
                               dbeta.data_ptr(), part.data_ptr(), nbytes, n, c, eps)
    else:
        ctx.rmsnorm_forward(x.data_ptr(), gamma.data_ptr(), y.data_ptr(), 0, n, c, eps, 0)
        ctx.rmsnorm_backward(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), dx.data_ptr(), dx.data_ptr(), dgamma.data_ptr(),
                             part.data_ptr(), nbytes, n, c, eps, 0)
    ctx.synchronize()
    X, D, Gm = _f64(x), _f64(dy), _f64(gamma)
    hh = X + _f64(r) if kind == "layer" else X
    mean = hh.mean(1, keepdim=True) if kind == "layer" else 0.0
    inv = 1.0 / torch.sqrt(((hh - mean) ** 2).mean(1, keepdim=True) + eps)
    want_y = (hh - mean) * inv * Gm + (_f64(beta) if kind == "layer" else 0.0)
    mean = X.mean(1, keepdim=True) if kind == "layer" else 0.0
    inv = 1.0 / torch.sqrt(((X - mean) ** 2).mean(1, keepdim=True) + eps)
    xh, dg = (X - mean) * inv, D * Gm
    want_dx = _f64(dres) + inv * (dg - (dg.mean(1, keepdim=True) if kind == "layer" else 0.0) - xh * (dg * xh).mean(1, keepdim=True))
    close = lambda a, b, tol: float(((a.double() - b).abs() / (b.abs() + b.square().mean().sqrt())).max()) < tol
    assert close(y[:n * c].view(n, c), want_y, 1e-5)
    if kind == "layer":
        assert torch.equal(h[:n * c].view(n, c), x + r)
        assert close(dbeta, 1.0 + D.sum(0), 1e-4)
    assert close(dx[:n * c].view(n, c), want_dx, 1e-4)
    assert close(dgamma, 1.0 + (D * xh).sum(0), 1e-4)
    for t in (y, dx):  # nothing is written behind the last element
        assert (t[n * c:] == 7.0).all()
    G.check_clean_status()


@pytest.mark.parametrize("c", [1026, 4095])
def test_backward_without_workspace(c):
    """The fixed workspace of this entry point may hold fewer partial rows than the launch would like."""
    ctx, _, _ = G.env()
    n = 3000
    g = torch.Generator(device="cuda")
    g.manual_seed(c)
    x, dy, gamma = (torch.randn(s, device="cuda", generator=g) for s in ((n, c), (n, c), (c,)))
    dx = torch.zeros(n, c, device="cuda")
    dgamma, dbeta = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    torch.cuda.synchronize()
    ctx.layernorm_backward_noalloc(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), 0, dx.data_ptr(), dgamma.data_ptr(),
                                   dbeta.data_ptr(), n, c, 1e-5)
    ctx.synchronize()
    X, D = x.double(), dy.double()
    inv = 1.0 / torch.sqrt(X.var(1, unbiased=False, keepdim=True) + 1e-5)
    xh, dg = (X - X.mean(1, keepdim=True)) * inv, D * gamma.double()
    want = inv * (dg - dg.mean(1, keepdim=True) - xh * (dg * xh).mean(1, keepdim=True))
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    assert rel(dx, want) < 1e-5 and rel(dgamma, (D * xh).sum(0)) < 1e-5 and rel(dbeta, D.sum(0)) < 1e-5
    G.check_clean_status()


# where the rules change hands, on the side of whole packets: element counts, even and odd lengths, packets per thread
BACKWARD = [(1963, 513), (1310, 769), (975, 1029), (870, 1151), (781, 1283), (657, 1537), (400, 2691), (300, 3331), (245, 4097),
            (80, 4101), (77, 5123), (90, 6145), (70, 6149), (66, 8191)]
EVEN = [(9800, 514, "rms"), (4300, 514, "layer"), (4900, 1026, "rms"), (2200, 1026, "layer"), (820, 2690, "layer"), (1230, 4098, "rms"),
        (540, 4098, "layer")]
FORWARD = [(3200, 258), (2500, 322), (1700, 486), (300, 4101), (297, 6530), (490, 8191), (500, 8191), (1400, 3002)]


@pytest.mark.parametrize("n,c,kind", [(n, c, k) for n, c in BACKWARD + FORWARD for k in ("layer", "rms")] + EVEN)
def test_norms_at_the_limits_of_whole_packets(n, c, kind):
    test_norms(n, c, 0, kind)
