"""Operand rows that a team of warps converts from registers: lengths where the team grows by a warp or its registers end,
with and without the channels being balanced, and a row count that leaves teams without a row.  The projection against
float64, relative to the sum of the sizes of a product's terms."""
import pytest
import torch

import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


def _rel(got, a, b):
    a, b = a.double(), b.double()
    return float(((got.double() - a @ b).abs() / (a.abs() @ b.abs())).max())


@pytest.mark.parametrize("power", [0, 30])
@pytest.mark.parametrize("n,k", [(4100, 640), (4100, 644), (3333, 1280), (3333, 1284), (1003, 2560), (1003, 2564), (515, 5120),
                                 (515, 5124)])
def test_row_lengths(n, k, power):
    ctx, _, _ = G.env()
    c = 1024
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    act, w, dout = (torch.randn(*s, device="cuda", generator=g) for s in ((n, k), (k, c), (n, c)))
    act[:, 3] *= 2.0 ** power
    w[3] *= 2.0 ** -power
    act[7] = 0
    out, dact, dw, db = (torch.zeros(*s, device="cuda") for s in ((n, c), (n, k), (k, c), (c,)))
    nbytes = ctx.linear_add_scratch_bytes(n, k, c, N.AG_CE_3XTF32)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    s = (scratch.data_ptr(), nbytes)
    ctx.linear_add_forward(0, act.data_ptr(), w.data_ptr(), 0, out.data_ptr(), n, k, c, N.AG_CE_3XTF32, *s)
    ctx.linear_add_backward(dout.data_ptr(), act.data_ptr(), w.data_ptr(), 0, dact.data_ptr(), dw.data_ptr(), db.data_ptr(),
                            n, k, c, N.AG_CE_3XTF32, *s)
    ctx.synchronize()
    G.check_clean_status()
    live = torch.arange(n, device="cuda") != 7
    assert bool((out[7] == 0).all())
    errs = _rel(out[live], act[live], w), _rel(dact, dout, w.T), _rel(dw, act.T, dout)
    print(f"{n} x {k} 2^{power}: " + " ".join("%.1e" % e for e in errs))
    assert errs[0] < 3e-6 and errs[1] < 1e-5 and errs[2] < 1e-5     # as for the other operand ranges
    # n terms in fp32, in 256 or fewer partial sums of 64 and more rows: n / 2 roundings of half an ulp at the very worst
    want, size = dout.double().sum(0), dout.double().abs().sum(0)
    assert bool(((db.double() - want).abs() <= n / 2 * 2.0 ** -24 * size).all())
