"""A method of the context that was replaced, on the class or on the object, is what a layer's launch goes through; what the
forms in Python took is taken by the compiled ones."""
import numpy as np
import pytest

import test_layer_calls as T
from autograd_b200 import _native as N
from autograd_b200.backend import _Layers
from autograd_b200.context import CudaContext

METHOD = {n: {"fill": "fill_f32"}.get(n, n) for n in T.LAYERS}

pytestmark = pytest.mark.skipif(not hasattr(N.calls, "layer_gelu_forward"), reason="the compiled module is not the binding here")


def _closed():
    """A context without a handle: whatever reaches the library is refused."""
    ctx = CudaContext.__new__(CudaContext)
    ctx._h, ctx._hi = None, 0
    return ctx


@pytest.mark.parametrize("where", ["class", "object", "dict"])
@pytest.mark.parametrize("name", T.LAYERS)
def test_a_replaced_method_is_called(name, where, monkeypatch):
    layer, args = getattr(N.calls, "layer_" + name), T._arguments(name, T._tensor((6, 8)))
    ctx, seen, want = _closed(), [], T._Recorder()

    def traced(*a, **kw):
        seen.append((METHOD[name], a[1:] if where == "class" else a, kw))

    if where == "class":
        monkeypatch.setattr(CudaContext, METHOD[name], traced)
    elif where == "object":
        setattr(ctx, METHOD[name], traced)
    else:
        ctx.__dict__[METHOD[name]] = traced
    layer(ctx, *args)
    getattr(_Layers, name)(want, *args)
    assert seen == want.calls
    if where != "class":
        other = _closed()
        with pytest.raises(N.AgError):
            layer(other, *args)
        delattr(ctx, METHOD[name])
    else:
        monkeypatch.undo()
    with pytest.raises(N.AgError):     # and no longer once it is back
        layer(ctx, *args)


def test_a_context_without_a_handle_attribute():
    ctx = CudaContext.__new__(CudaContext)
    for name in T.LAYERS:
        with pytest.raises(AttributeError):
            getattr(N.calls, "layer_" + name)(ctx, *T._arguments(name, T._tensor((6, 8))))


@pytest.mark.parametrize("value", ["0.5", np.float64(0.5), np.array(0.5), True, 7])
def test_values_that_fills_take(value):
    """Whatever float() makes a number of."""
    storage = T._tensor((4,)).storage
    with pytest.raises(N.AgError):     # the library's refusal of the null handle: the value was taken
        N.calls.layer_fill(_closed(), storage, value)
    with pytest.raises((TypeError, ValueError)):
        N.calls.layer_fill(_closed(), storage, "half")


@pytest.mark.parametrize("name", ["swiglu_forward", "swiglu_backward"])
def test_a_row_of_gate_and_up_may_have_more_elements_than_an_int(name):
    """It is the half of it that has to fit."""
    layer = getattr(N.calls, "layer_" + name)
    t = T._tensor((1, 3 << 30), np.uint16)
    with pytest.raises(N.AgError):     # the library's refusal of the null handle
        layer(_closed(), t, t)
    t = T._tensor((1, 1 << 32), np.uint16)
    with pytest.raises(OverflowError):
        layer(_closed(), t, t)
