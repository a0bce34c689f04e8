"""Projections of few columns over many rows, which go straight from fp32 operands whatever their length, and the sizes beside
the limits of that rule, where forward and backward may take different paths.  Against float64, relative to the sum of the sizes
of a product's terms."""
import pytest
import torch

import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu

# a product errs by 2^-22 or 2^-8 of the sizes of its terms at most, chains and splits by less; backward adds to zero
BOUND = {N.AG_CE_3XTF32: 3e-6, N.AG_CE_BF16: 2.0 ** -7}


def _rel(got, a, b, extra=None):
    a, b = a.double(), b.double()
    want, size = a @ b, a.abs() @ b.abs()
    if extra is not None:
        want, size = want + extra, size + extra.abs()
    return float(((got.double() - want).abs() / size).max())


@pytest.mark.parametrize("precision", list(BOUND))
@pytest.mark.parametrize("n,k,c", [(16384, 3312, 88), (9001, 5120, 128), (30011, 1032, 64), (70000, 520, 136), (73729, 264, 40),
                                   (16384, 3312, 192),     # forward on operand pairs, backward not
                                   (8003, 1024, 384), (3001, 5120, 384), (4001, 36000, 32), (2001, 36872, 32)])
def test_projection(n, k, c, precision):
    ctx, _, _ = G.env()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    act, w, dout, x, b = (torch.randn(*s, device="cuda", generator=g) for s in ((n, k), (k, c), (n, c), (n, c), (c,)))
    out, dx, dact, dw, db = (torch.zeros(*s, device="cuda") for s in ((n, c), (n, c), (n, k), (k, c), (c,)))
    nbytes = ctx.linear_add_scratch_bytes(n, k, c, precision)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    p = [t.data_ptr() for t in (x, act, w, b, out, dout, dx, dact, dw, db)]
    s = (scratch.data_ptr(), nbytes)
    ctx.linear_add_forward(*p[:5], n, k, c, precision, *s)
    ctx.linear_add_backward(p[5], p[1], p[2], *p[6:], n, k, c, precision, *s)
    ctx.synchronize()
    G.check_clean_status()
    errs = (_rel(out, act, w, x.double() + b.double()), _rel(dact, dout, w.T), _rel(dw, act.T, dout))
    print(f"{n} x {k} x {c}: " + " ".join("%.1e" % e for e in errs))
    assert max(errs) < BOUND[precision]
    assert torch.equal(dx, dout)
