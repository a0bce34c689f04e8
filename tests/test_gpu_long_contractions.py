"""bf16 products over very many rows: the tensor core's accumulator truncates, so that the error grows with the length of
one accumulation chain, which therefore has to be bounded.  Operands that bf16 holds exactly, all of one sign (nothing
averages out), against float64."""
import pytest
import torch

import gpu_util as G
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu

CHAIN = 8192    # elements of one chain at most
# A chain is CHAIN / 16 MMAs.  Each adds its 16 products in at most two steps that cut off less than an ulp (2^-23 of the
# sum so far); the sum grows evenly, so half of the final sum on average.  Adding up chains and partial outputs (round
# to nearest) stays below an eighth of that.
BOUND = CHAIN / 16 * 2 * 2.0 ** -23 / 2 * 1.125


def _exact(rows, cols, seed):
    """bf16 values in [1, 2)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (1 + torch.randint(0, 128, (rows, cols), device="cuda", generator=g, dtype=torch.int32) / 128).float()


@pytest.mark.parametrize("rows,k,c", [(1 << 21, 64, 64), ((1 << 19) + 77, 128, 96), (CHAIN, 64, 64), (CHAIN + 1, 64, 64)])
def test_weight_gradient_of_many_rows(rows, k, c):
    ctx, _, _ = G.env()
    act, dout = _exact(rows, k, 1), _exact(rows, c, 2)
    dw = torch.zeros(k, c, device="cuda")
    nbytes = ctx.linear_add_scratch_bytes(rows, k, c, N.AG_CE_BF16)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.linear_add_backward(dout.data_ptr(), act.data_ptr(), 0, 0, 0, dw.data_ptr(), 0, rows, k, c, N.AG_CE_BF16,
                            scratch.data_ptr(), nbytes)
    ctx.synchronize()
    G.check_clean_status()
    want = torch.zeros(k, c, device="cuda", dtype=torch.float64)
    for r in range(0, rows, 1 << 18):
        want += act[r:r + (1 << 18)].double().T @ dout[r:r + (1 << 18)].double()
    err = float(((dw.double() - want).abs() / want).max())
    print(f"dW over {rows} rows: {err:.2e} (bound {BOUND:.2e})")
    assert err < BOUND


def test_projection_with_a_long_inner_dimension():
    rows, k, c = 128, 1 << 17, 64
    ctx, _, _ = G.env()
    act, w = _exact(rows, k, 3), _exact(k, c, 4)
    out = torch.zeros(rows, c, device="cuda")
    nbytes = ctx.linear_add_scratch_bytes(rows, k, c, N.AG_CE_BF16)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.linear_add_forward(0, act.data_ptr(), w.data_ptr(), 0, out.data_ptr(), rows, k, c, N.AG_CE_BF16,
                           scratch.data_ptr(), nbytes)
    ctx.synchronize()
    G.check_clean_status()
    want = act.double() @ w.double()
    err = float(((out.double() - want).abs() / want).max())
    print(f"forward over {k} elements: {err:.2e} (bound {BOUND:.2e})")
    assert err < BOUND
