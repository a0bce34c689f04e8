"""The compiled calls of the backend's layers: any other context goes through the forms in Python, with the same arguments, and
what those refuse stays refused."""
import types

import numpy as np
import pytest

from autograd_b200 import _native as N
from autograd_b200 import hostgraph as hg
from autograd_b200.backend import _Layers
from autograd_b200.context import CudaContext

LAYERS = [n for n in vars(_Layers) if not n.startswith("_")]


class _Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args, **kw: self.calls.append((name, args, kw))


def _tensor(shape, dtype=np.float32):
    t = hg.HostTensor(shape, dtype, requires_grad=False)
    t.storage = types.SimpleNamespace(shape=shape, dtype=dtype, nbytes=0, ptr=types.SimpleNamespace(buffer_id=4096, offset=16))
    return t


def _arguments(name, t):
    s = t.storage
    return {"gelu_forward": (t, t), "gelu_backward": (t, t, t), "add_layernorm_forward": (t, None, t, t, t, t, None, None, 1e-5),
            "rmsnorm_forward": (t, t, t, None, 1e-6), "swiglu_forward": (t, t), "swiglu_backward": (t, t),
            "rope_qk": (t, None, t, t, 2, 3, 4, 0, 8, 1, 0), "fill": (s, 0.0),
            "adamw_step": (s, s, s, s, 1e-3, 1e-3, 0.9, 0.95, 1e-8, 0.1, 1.0)}[name]


@pytest.mark.parametrize("dtype", [np.float32, np.dtype(np.float32), np.uint16])
@pytest.mark.parametrize("name", LAYERS)
def test_other_contexts_get_the_calls_of_the_python_forms(name, dtype):
    layer = getattr(N.calls, "layer_" + name, None)
    if layer is None:
        pytest.skip("the compiled module is not the binding here")
    args = _arguments(name, _tensor((6, 8), dtype))
    one, two = _Recorder(), _Recorder()
    layer(one, *args)
    getattr(_Layers, name)(two, *args)
    assert one.calls == two.calls and len(one.calls) == 1
    with pytest.raises(TypeError):
        layer(one, *args, 0)


def test_without_a_handle_there_is_an_error():
    """A closed context: the library refuses the null handle, as it does through the context's own methods."""
    if not hasattr(N.calls, "layer_gelu_forward"):
        pytest.skip("the compiled module is not the binding here")
    closed = CudaContext.__new__(CudaContext)
    closed._h, closed._hi = None, 0
    for name in LAYERS:
        with pytest.raises(N.AgError):
            getattr(N.calls, "layer_" + name)(closed, *_arguments(name, _tensor((6, 8))))
    with pytest.raises(IndexError):
        N.calls.layer_rmsnorm_forward(closed, *_arguments("rmsnorm_forward", _tensor(())))
    with pytest.raises(TypeError):
        N.calls.layer_fill(closed, _tensor((4,), np.complex64).storage, 0.0)
