"""LayerNorm / RMSNorm where a team of warps takes a row: few rows, and row lengths without 16-byte packets.  Sizes at
the edges of the team shapes, against the oracle."""
import numpy as np
import pytest

import gpu_util as G
from autograd_b200 import _native as N
from conftest import TOL_BF16, TOL_BWD, TOL_FWD, assert_close
from oracle import fused_layers as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1280), (8, 1280), (296, 1536), (297, 1026), (5, 77), (600, 255), (33, 2049), (3, 4099), (7, 1), (2, 8190),
          (4000, 62), (1200, 513), (130, 4096), (2, 2050), (70, 1537)]


def _addr(t):
    return t.storage.ptr.address


@pytest.mark.parametrize("n,c", SHAPES)
def test_layernorm_teams_vs_oracle(n, c):
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(n * 7 + c)
    x, r, dy = (rng.standard_normal((n, c), dtype=np.float32) for _ in range(3))
    gam, bet = 1 + 0.1 * rng.standard_normal(c, dtype=np.float32), 0.1 * rng.standard_normal(c, dtype=np.float32)
    X, R, GM, BT = G.up(x), G.up(r), G.up(gam), G.up(bet)
    H, Y = G.empty((n, c)), G.empty((n, c))
    MEAN, RSTD = G.empty((n,)), G.empty((n,))
    ctx.add_layernorm_forward(_addr(X), _addr(R), _addr(GM), _addr(BT), _addr(H), _addr(Y), _addr(MEAN), _addr(RSTD), n, c, 1e-5)
    h = x + r
    assert np.array_equal(G.down(H), h)
    assert_close(G.down(Y), O.layernorm_forward(h, gam, bet, 1e-5)[0], TOL_FWD, "y")
    assert_close(G.down(RSTD), 1 / np.sqrt(h.astype(np.float64).var(axis=1) + 1e-5), TOL_FWD, "rstd")
    DY, DX = G.up(dy), G.up(r)
    DG, DB = G.up(np.zeros(c, np.float32)), G.up(np.zeros(c, np.float32))
    part = G.empty((ctx.norm_partials_bytes(c) // 4,))
    ctx.layernorm_backward(_addr(DY), _addr(H), _addr(GM), _addr(DX), _addr(DX), _addr(DG), _addr(DB), _addr(part),
                           ctx.norm_partials_bytes(c), n, c, 1e-5)
    zero = np.zeros(c, np.float32)
    dx, dg, db = O.layernorm_backward(h, gam, dy, 1e-5, r, zero, zero)
    if c > 1:  # one column: dx is rounding only
        assert_close(G.down(DX), dx, TOL_BWD, "dx")
    assert_close(G.down(DG), dg, TOL_BWD, "dgamma") if c > 1 else None
    assert_close(G.down(DB), db, TOL_BWD, "dbeta")
    G.check_clean_status()
    G.free(X, R, GM, BT, H, Y, MEAN, RSTD, DY, DX, DG, DB, part)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n,c", [s for s in SHAPES if s[1] > 1])
def test_rmsnorm_teams_vs_oracle(n, c, dtype):
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(n * 11 + c)
    bf = dtype == "bf16"
    x, dz, res = (rng.standard_normal((n, c), dtype=np.float32) for _ in range(3))
    if bf:
        x, dz, res = (O.round_to_bf16(a) for a in (x, dz, res))
    gam = 1 + 0.1 * rng.standard_normal(c, dtype=np.float32)
    up = (lambda a: G.up(O.f32_to_bf16_bits(a))) if bf else G.up
    X, DZ, RES, GM = up(x), up(dz), up(res), G.up(gam)
    Y, DX = (G.empty((n, c), dtype=np.uint16 if bf else np.float32) for _ in range(2))
    DG = G.up(np.zeros(c, np.float32))
    part = G.empty((ctx.norm_partials_bytes(c) // 4,))
    dt = N.AG_BF16 if bf else N.AG_F32
    ctx.rmsnorm_forward(_addr(X), _addr(GM), _addr(Y), 0, n, c, 1e-6, dt)
    ctx.rmsnorm_backward(_addr(DZ), _addr(X), _addr(GM), _addr(RES), _addr(DX), _addr(DG), _addr(part),
                         ctx.norm_partials_bytes(c), n, c, 1e-6, dt)
    down = (lambda t: O.bf16_bits_to_f32(G.down_bits(t))) if bf else G.down
    dx, dg = O.rmsnorm_backward(x, gam, dz, 1e-6, res, np.zeros(c, np.float32))
    assert_close(down(Y), O.rmsnorm_forward(x, gam, 1e-6)[0], TOL_BF16 if bf else TOL_FWD, "y")
    assert_close(down(DX), dx, TOL_BF16 if bf else TOL_BWD, "dx")
    assert_close(G.down(DG), dg, TOL_BWD, "dgamma")
    G.check_clean_status()
    G.free(X, DZ, RES, GM, Y, DX, DG, part)
