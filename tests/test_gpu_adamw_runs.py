"""Rows of AdamW launches: those on memory apart overlap, those that share memory, or that follow other work on the
stream, must not.  Sizes around a packet, a CTA and a resident wave."""
import numpy as np
import pytest

import gpu_util as G
from conftest import TOL_FWD, assert_close
from oracle import fused_layers as O

pytestmark = pytest.mark.gpu

HP = (1e-2, 9e-3, 0.9, 0.95, 1e-8, 0.1)
# around one packet, one CTA of 256 packets, and a wave of 148 SMs x 3 CTAs (one and two packets per thread)
SIZES = [1, 3, 4, 5, 1023, 1024, 1025, 454_655, 454_660, 909_313, 3_000_001]


def _oracle(state, g, bf16):
    if bf16:
        return list(O.adamw_step_bf16grad(state[0], g, state[1], state[2], *HP))
    return list(O.adamw_step(state[0], g, state[1], state[2], *HP))


@pytest.mark.parametrize("bf16", [False, True])
def test_rows_of_steps_match_oracle(bf16):
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(3)
    params = []
    for n in SIZES * 3:
        p, m = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
        v = rng.random(n).astype(np.float32)
        g = rng.standard_normal(n).astype(np.float32)
        if bf16:
            g = (g.view(np.uint32) >> 16).astype(np.uint16)
        params.append(([p, m, v], g, [G.up(x) for x in (p, g, m, v)]))
    for _ in range(3):
        for state, g, (p, gr, m, v) in params:
            be.adamw_step(p.storage, gr.storage, m.storage, v.storage, None, *HP)
    for state, g, dev in params:
        for _ in range(3):
            state = _oracle(state, g, bf16)
        for what, d, ref in zip("pmv", (dev[0], dev[2], dev[3]), state):
            assert_close(G.down(d), ref, TOL_FWD, f"{what} of {g.size}")
        G.free(*dev)


@pytest.mark.parametrize("n", [1000, 3_000_001])
def test_steps_on_shared_memory_keep_their_order(n):
    """The same parameter twice; the gradient of one step is the parameter of the one before; a copy between two."""
    ctx, alloc, be = G.env()
    rng = np.random.default_rng(4)
    a, b = ([rng.random(n).astype(np.float32) for _ in range(3)] for _ in range(2))
    g = rng.standard_normal(n).astype(np.float32)
    da, db = ([G.up(x) for x in s] for s in (a, b))
    dg = G.up(g)

    def step(s, grad):
        be.adamw_step(s[0].storage, grad.storage, s[1].storage, s[2].storage, None, *HP)

    for _ in range(4):
        step(da, dg)
        step(da, dg)
        step(db, da[0])
        be.copy_from_host(dg, b[0])
        step(da, dg)
        be.copy_from_host(dg, g)
    b0 = b[0]
    for _ in range(4):
        a = _oracle(_oracle(a, g, False), g, False)
        b = _oracle(b, a[0], False)
        a = _oracle(a, b0, False)
    for what, d, ref in zip(("a.p", "a.m", "a.v", "b.p", "b.m", "b.v"), da + db, a + b):
        assert_close(G.down(d), ref, TOL_FWD * 10, what)
    G.free(dg, *da, *db)
