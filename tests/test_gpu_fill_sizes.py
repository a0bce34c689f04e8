"""Fills on both sides of the sizes where the kernel takes over from the memset, at unaligned starts, exact to the word."""
import numpy as np
import pytest

import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, (1 << 21) - 1, 1 << 21, (1 << 21) + 3, 1 << 24, (1 << 24) + 1])
@pytest.mark.parametrize("value", [0.0, -2.5])
@pytest.mark.parametrize("start", [0, 1, 3])
def test_fill_writes_its_words_only(n, value, start):
    ctx, alloc, be = G.env()
    guard = np.arange(1, 9, dtype=np.float32)
    st = alloc.alloc((start + n + 8,), np.float32)
    at = st.ptr.address
    ctx.fill_f32(at, 7.0, start + n)
    ctx.copy_from_host(at + 4 * (start + n), guard)
    ctx.fill_f32(at + 4 * start, value, n)
    got = ctx.copy_to_host(at, (start + n + 8,), np.float32)
    assert np.all(got[:start] == 7.0) and np.array_equal(got[start + n:], guard)
    assert np.all(got[start:start + n] == value)
    ctx.synchronize()
    alloc.free(st)
