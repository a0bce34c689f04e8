"""What a launch takes where it wants an address: an int, None, a tensor, a tensor without storage, a storage."""
import numpy as np
import pytest

from autograd_b200 import _native as N
from autograd_b200 import hostgraph as hg
from autograd_b200.storage import CudaMemPointer, Storage


def _tensor(address, offset=0, shape=(3, 4)):
    t = hg.HostTensor(shape)
    t.storage = Storage(CudaMemPointer(address, offset), shape, np.float32, "cuda", 48)
    return t


@pytest.mark.parametrize("compiled", [True, False])
def test_address_arguments(compiled):
    """A context that is null fails every call before anything is touched: the arguments have been converted by then."""
    calls = N.calls if compiled else N._CheckedCalls(N.lib)
    t = _tensor(1 << 40, 256)
    for a in (0, None, 1 << 40, np.int64(1 << 40), t, t.storage, hg.HostTensor((3,))):
        with pytest.raises(N.AgError):
            calls.ag_gelu_forward(0, a, t, 12)
    for a in ("x", object(), 1.5j):
        with pytest.raises((TypeError, ValueError, AttributeError)):
            calls.ag_gelu_forward(0, a, t, 12)


def test_questions_of_a_tensor():
    from autograd_b200 import backend as B
    t = _tensor(1 << 40, 256, (2, 3, 4))
    assert B._addr(t) == (1 << 40) + 256 and B._addr(None) == 0 and B._addr(hg.HostTensor((3,))) == 0
    assert B._rows_cols(t) == (6, 4) and B._size(t) == 24 and B._size(hg.HostTensor(())) == 1
    with pytest.raises(IndexError):
        B._rows_cols(hg.HostTensor(()))
    with pytest.raises((AttributeError, TypeError)):
        B._addr(object())
