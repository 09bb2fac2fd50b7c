"""The order of steps that run on different streams, from the calls that the models make: no GPU."""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from pygpukit_b200.core import stream as streams
from pygpukit_b200.llm.models import causal


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append(name)


@pytest.fixture
def model(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(causal, "api", rec)
    monkeypatch.setattr(causal, "is_capturing", lambda h: h is not None and h in capturing, raising=False)
    capturing = []
    m = object.__new__(causal.CausalTransformerModel)
    m._last_stream, m._num_sequences, m.comm, m.blocks = None, 1, None, []
    array = SimpleNamespace(device_ptr=64, shape=(1, 8), slice_rows=lambda n: array)
    m._buffers = SimpleNamespace(state_buf=array, next_token=array, hidden=array, token_buf=array)
    m._graph_stream = SimpleNamespace(handle=object())
    m._graph = SimpleNamespace(replay=lambda s: rec.calls.append("replay"))
    m._pinned_state = lambda: (C.c_void_p(64), np.zeros(4, np.int32))
    m._embed_rows = lambda *a: rec.calls.append("embed")
    m.rec, m.capturing = rec, capturing
    return m


def calls(m):
    out, m.rec.calls = m.rec.calls, []
    return out


def test_a_step_waits_for_the_last_one_on_another_stream(model):
    """Prompts run on the caller's stream and do not wait for their end, captured steps on a stream of their own: each change of stream
    waits before the shared arrays are touched, and steps on one stream never wait."""
    m = model
    m._embed([1], 1, 0, m._buffers)
    assert calls(m) == ["device_sync", "upload", "embed"]
    m._embed([1], 1, 0, m._buffers)
    assert calls(m) == ["upload", "embed"]
    m.decode_step_host(5, 1)
    assert calls(m) == ["device_sync", "memcpy_h2d", "replay", "memcpy_d2h", "stream_sync"]
    m.decode_step_host(5, 2)
    m.decode_graph_replay()
    assert "device_sync" not in calls(m)
    m.set_decode_state(3, 4)
    got = calls(m)
    assert got.index("device_sync") < got.index("memcpy_h2d")
    m.decode_graph_replay()
    assert calls(m) == ["device_sync", "replay"]
    m._embed([1], 1, 0, m._buffers)
    assert calls(m) == ["device_sync", "upload", "embed"]


def test_a_recorded_step_neither_waits_nor_counts(model):
    m, side = model, SimpleNamespace(handle=object())
    m._embed([1], 1, 0, m._buffers)
    calls(m)
    m.capturing.append(side.handle)
    with streams.use_stream(side):
        m._enter(streams.current_stream_handle())
    assert calls(m) == []
    m._embed([1], 1, 0, m._buffers)
    assert calls(m) == ["upload", "embed"]


def test_work_left_open_is_waited_for_when_the_stream_changes(monkeypatch):
    """A replayed decode step is not waited for on its own stream, and complete for everyone else: a change of the current stream, in
    either direction, and a capture wait for it -- once, and not where nothing was left open."""
    log = []

    class Api:
        def __getattr__(self, name):
            return lambda *a: log.append((name, *a[:1]))

    monkeypatch.setattr(streams, "api", Api())
    s, t = SimpleNamespace(handle=object()), SimpleNamespace(handle=object())
    with streams.use_stream(s):
        pass
    assert log == []
    streams.leave_open()
    with streams.use_stream(None):
        assert log == []
        with streams.use_stream(s):
            assert log == [("stream_sync", None)]
            streams.leave_open()
            with streams.use_stream(s):
                assert len(log) == 1
            with streams.use_stream(t):
                assert log[1:] == [("stream_sync", s.handle)]
            streams.leave_open()
        assert log[2:] == [("stream_sync", s.handle)]
    assert len(log) == 3
    with streams.use_stream(s):
        streams.leave_open()
        with streams.CudaGraph().capture(s):
            assert log[3:] == [("stream_sync", s.handle), ("graph_begin", s.handle)]
    assert log[5] == ("graph_end", s.handle)


def test_a_wait_that_fails_leaves_the_right_stream_current(monkeypatch):
    def fail(*a):
        raise RuntimeError("ran out")

    monkeypatch.setattr(streams, "api", SimpleNamespace(stream_sync=fail))
    s = SimpleNamespace(handle=object())
    streams.leave_open()
    with pytest.raises(RuntimeError, match="ran out"):
        with streams.use_stream(s):
            raise AssertionError("not entered")
    assert streams.current_stream_handle() is None
    with pytest.raises(RuntimeError, match="ran out"):
        with streams.use_stream(s):
            streams.leave_open()
    assert streams.current_stream_handle() is None and not streams._open
