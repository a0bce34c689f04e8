"""Memory that a step takes only to save time: none where little is left, none after an allocation that fails for want of
memory, as much as the configuration allows otherwise; any other error of an allocation is one."""
import pytest

from autograd_b200 import _native as N
from autograd_b200.context import CudaContext
from autograd_b200.step import FusedLayerStep, StepConfig
from autograd_b200.storage import CudaAllocator

PARTIALS, LOGITS, TOTAL = 12345, 7 << 20, 1 << 32
CFG = dict(n_layer=3, n_embd=32, n_head=1, head_dim=32, seq_len=8, vocab=64, batch=1)


class _Device:
    eager, sm_count = False, 148
    flce_desc = staticmethod(CudaContext.flce_desc)

    def __init__(self, free=TOTAL, refuse=(), error=None):
        self.free_bytes, self.refuse, self.error, self.live = free, refuse, error, {}

    def memory(self):
        return self.free_bytes, TOTAL

    def alloc(self, nbytes):
        if nbytes in self.refuse:
            raise self.error
        self.free_bytes -= nbytes
        if self.free_bytes < 0:
            raise N.AgError(N.AG_ERR_CUDA, f"cudaMalloc of {nbytes} bytes failed: out of memory")
        at = (len(self.live) + 1) << 32
        self.live[at] = nbytes
        return at

    def norm_partials_bytes(self, c):
        return PARTIALS

    scatter_add_scratch_bytes = flce_scratch_bytes = lambda self, *a: 1 << 20

    def flce_logits_bytes(self, desc):
        return LOGITS

    def __getattr__(self, name):
        return lambda *a, **k: None


def _step(device, **cfg):
    return FusedLayerStep(device, CudaAllocator(device), None, StepConfig(**CFG, **cfg))


def _needed():
    d = _Device()
    _step(d, logits_max_bytes=0, partials_max_bytes=0)
    return sum(d.live.values())


def test_what_the_configuration_allows():
    st = _step(_Device())
    assert st._batch == 7 and st.logits_bytes == LOGITS and st._keeps()
    st = _step(_Device(), logits_max_bytes=LOGITS - 1, partials_max_bytes=3 * PARTIALS + 1)
    assert st._batch == 3 and st.logits is None and st.logits_bytes == 0 and not st._keeps()
    st = _step(_Device(), logits_max_bytes=LOGITS, partials_max_bytes=0)
    assert st._batch == 1 and st.logits_bytes == LOGITS


@pytest.mark.parametrize("left,batch,logits", [(0, 1, 0), ((TOTAL >> 4) + 6 * PARTIALS - 1, 1, 0),
                                               ((TOTAL >> 4) + 6 * PARTIALS, 7, 0),
                                               ((TOTAL >> 4) + 6 * PARTIALS + LOGITS, 7, LOGITS)])
def test_little_memory(left, batch, logits):
    """A step that just fits is made, and what it can do without leaves a sixteenth of the device."""
    st = _step(_Device(free=_needed() + left))
    assert (st._batch, st.logits_bytes) == (batch, logits)


@pytest.mark.parametrize("refuse,batch,logits", [(7 * PARTIALS, 1, LOGITS), (LOGITS, 7, 0)])
@pytest.mark.parametrize("error", [MemoryError(), N.AgError(N.AG_ERR_CUDA, "cudaMalloc failed: out of memory")])
def test_an_allocation_that_fails(refuse, batch, logits, error):
    st = _step(_Device(refuse=(refuse,), error=error))
    assert (st._batch, st.logits_bytes) == (batch, logits) and st._keeps() == (logits > 0)


@pytest.mark.parametrize("refuse", [7 * PARTIALS, LOGITS])
def test_other_errors_are_errors(refuse):
    with pytest.raises(N.AgError, match="illegal"):
        _step(_Device(refuse=(refuse,), error=N.AgError(N.AG_ERR_CUDA, "an illegal memory access was encountered")))
