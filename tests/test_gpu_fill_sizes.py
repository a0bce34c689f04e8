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


@pytest.mark.parametrize("n", [1, 2, 3, 7, 64, 1001])
@pytest.mark.parametrize("start", [0, 1, 2, 7])
def test_zero_fill_of_16_bit_words(n, start):
    """Cleared in words of 32 bits where the start and the length allow it."""
    ctx, alloc, be = G.env()
    st = alloc.alloc((start + n + 8,), np.uint16)
    at = st.ptr.address
    ctx.fill_pattern(at, 0x1234, 2, start + n + 8)
    ctx.fill_pattern(at + 2 * start, 0, 2, n)
    got = ctx.copy_to_host(at, (start + n + 8,), np.uint16)
    assert np.all(got[:start] == 0x1234) and np.all(got[start:start + n] == 0) and np.all(got[start + n:] == 0x1234)
    alloc.free(st)
