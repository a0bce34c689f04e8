"""When a step records its launches: not while the program captures the stream, and an error of the recording is no error
of the step.  The device is a stand-in that counts what reaches it."""
import pytest

from autograd_b200 import _native as N
from autograd_b200.step import FamilyTimer, FusedLayerStep


class _Device:
    eager = False

    def __init__(self):
        self.fail = []        # error codes of the recordings to come, None: it succeeds
        self.log = []

    def record(self, fn):
        code = self.fail.pop(0) if self.fail else None
        if code is not None:
            self.log.append("refused")
            raise N.AgError(code, "recording failed")
        self.log.append("recorded")
        return len(self.log)

    def replay(self, graph):
        self.log.append("replayed")

    def drop_recording(self, graph):
        self.log.append("dropped")


def _step(device):
    st = FusedLayerStep.__new__(FusedLayerStep)
    st.ctx, st.desc, st.timer, st._small = device, b"first", FamilyTimer(device), True
    st._graph = st._graph_key = st._stepped = st._unrecordable = None
    st.forward = lambda: device.log.append("launched")
    st.backward = lambda: None
    return st


def _run(st, device, steps=1):
    del device.log[:]
    for _ in range(steps):
        st.step()
    return device.log


def test_a_step_captured_after_one_warm_up_step_is_launched_and_recorded_later():
    device = _Device()
    st = _step(device)
    assert _run(st, device) == ["launched"]
    device.fail = [N.AG_ERR_CAPTURING, N.AG_ERR_CAPTURING]
    assert _run(st, device, 2) == ["refused", "launched"] * 2
    assert _run(st, device, 2) == ["recorded", "launched", "replayed"]


@pytest.mark.parametrize("code", [N.AG_ERR_CUDA, N.AG_ERR_INVALID])
def test_a_recording_that_fails_is_not_tried_again(code):
    device = _Device()
    st = _step(device)
    _run(st, device)
    device.fail = [code]
    assert _run(st, device, 3) == ["refused", "launched", "launched", "launched"]
    st.desc = b"second"       # other launches: they may be recordable
    assert _run(st, device, 3) == ["launched", "recorded", "launched", "replayed"]


def test_the_old_recording_goes_only_once_there_is_a_new_one():
    """Dropping one waits for the stream, which a program that captures it cannot have."""
    device = _Device()
    st = _step(device)
    assert _run(st, device, 3) == ["launched", "recorded", "launched", "replayed"]
    st.desc = b"second"
    _run(st, device)
    device.fail = [N.AG_ERR_CAPTURING]
    assert _run(st, device) == ["refused", "launched"]
    assert _run(st, device) == ["recorded", "dropped", "launched"]
