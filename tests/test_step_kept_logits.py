"""Whose logits a step's buffer holds between forward and backward: under descriptors in turn, beside replayed steps and after
calls that fail.  The device is a stand-in that remembers which descriptor and batch wrote the buffer last."""
import pytest

from autograd_b200 import _native as N
from autograd_b200.context import CudaContext
from autograd_b200.step import FusedLayerStep, StepConfig
from autograd_b200.storage import CudaAllocator


class _Device:
    """Launches take effect at once; those of a recording at each replay."""
    eager, sm_count = False, 148
    flce_desc = staticmethod(CudaContext.flce_desc)

    def __init__(self):
        self.next, self.inside, self.batch = 1 << 28, None, 0     # inside: (descriptor, batch) of the logits in the buffer
        self.effects, self.log, self.fail = None, [], {}          # fail: method -> exception

    def alloc(self, nbytes):
        self.next += (int(nbytes) + 255) // 256 * 256
        return self.next

    def memory(self):
        return 1 << 36, 1 << 37

    norm_partials_bytes = scatter_add_scratch_bytes = flce_scratch_bytes = lambda self, *a: 4096

    def flce_logits_bytes(self, desc):
        return 0 if desc.precision == N.AG_CE_FP32 else 1 << 16

    def _do(self, effect):
        if self.effects is None:
            effect()
        else:
            self.effects.append(effect)

    def _check(self, name):
        if name in self.fail:
            raise self.fail.pop(name)

    def flce_forward_keep(self, desc, *a):
        self._check("flce_forward_keep")
        key = bytes(desc)
        self._do(lambda: setattr(self, "inside", (key, self.batch)))

    def flce_backward_kept(self, desc, *a):
        key = bytes(desc)

        def read():
            assert self.inside == (key, self.batch)
            self.log.append("kept")
        self._do(read)

    def flce_backward(self, *a):
        self._do(lambda: self.log.append("recomputed"))

    def layernorm_backward_rows(self, *a):
        self._check("layernorm_backward_rows")

    def record(self, fn):
        self.effects = effects = []
        try:
            fn(self)
            self._check("record")
        finally:
            self.effects = None
        return effects

    def replay(self, graph):
        self._check("replay")
        for effect in graph:
            effect()

    def __getattr__(self, name):
        return lambda *a, **k: None


def _step():
    d = _Device()
    cfg = StepConfig(n_layer=1, n_embd=32, n_head=1, head_dim=32, seq_len=8, vocab=64, batch=1)
    st = FusedLayerStep(d, CudaAllocator(d), None, cfg)
    others = [d.flce_desc(st.N, st.C, st.V, precision=p) for p in (N.AG_CE_BF16X3, N.AG_CE_FP32)]
    return d, st, st.desc, others


def _replaying():
    d, st, a, others = _step()
    for _ in range(3):
        st.step()
    assert st._graph is not None and d.log == ["kept"] * 3
    d.log.clear()
    return d, st, a, others


def test_a_forward_that_fails_leaves_no_logits_behind():
    d, st, a, _ = _step()
    st.forward()
    d.batch = 1
    d.fail["flce_forward_keep"] = N.AgError(N.AG_ERR_SCRATCH, "refused")
    with pytest.raises(N.AgError):
        st.forward()
    st.backward()
    st.forward()
    st.backward()
    assert d.log == ["recomputed", "kept"]


def test_a_replayed_step_takes_the_buffer_over():
    """forward() under one descriptor, a replayed step under another one, backward() under the first, and the other way round."""
    d, st, a, (b, _) = _replaying()
    st.desc = b
    st.forward()
    st.desc, d.batch = a, 1
    st.step()
    assert d.log == ["kept"]
    st.desc = b
    st.backward()
    st.desc = a
    st.backward()
    assert d.log == ["kept", "recomputed", "kept"]


def test_descriptors_in_turn():
    d, st, a, (b, exact) = _step()
    for fwd, bwd, want in ((a, a, "kept"), (a, b, "recomputed"), (b, a, "recomputed"), (exact, a, "recomputed"),
                           (b, b, "kept"), (a, exact, "recomputed"), (exact, exact, "recomputed")):
        st.desc = fwd
        st.forward()
        st.desc = bwd
        st.backward()
        assert d.log.pop() == want


@pytest.mark.parametrize("where", ["layernorm_backward_rows", "record", "replay"])
def test_a_recording_or_replay_that_fails(where):
    d, st, a, (b, _) = _step()
    if where == "replay":
        d, st, a, (b, _) = _replaying()
    else:
        st.step()
    d.log.clear()
    st.desc = b
    st.forward()
    st.desc, d.batch = a, 1
    d.fail[where] = KeyError("an error that is no refusal") if where != "replay" else N.AgError(N.AG_ERR_CUDA, "failed")
    with pytest.raises((KeyError, N.AgError)):
        st.step()
    st.desc, d.batch = b, 0      # a recording has run nothing
    st.backward()
    assert d.log == ["kept" if where != "replay" else "recomputed"]


def test_a_new_recording_that_fails_leaves_the_old_one_its_logits():
    d, st, a, (b, _) = _replaying()
    st.desc = b
    st.step()
    d.fail["record"] = N.AgError(N.AG_ERR_CUDA, "failed")
    st.step()
    st.desc, d.batch = a, 2
    st.step()
    st.backward()
    assert d.log == ["kept"] * 4
