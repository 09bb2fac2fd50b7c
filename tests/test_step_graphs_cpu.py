"""Which captured decode steps a layered model keeps, from the calls that it makes: no GPU."""
from types import SimpleNamespace

import numpy as np
import pytest

from pygpukit_b200.llm import paged_cache
from pygpukit_b200.llm.models import layered


class Array:
    """a device array whose memory comes back at the address it had"""

    def __init__(self, shape, dtype=None):
        self.shape, self.size, self.device_ptr, self.nbytes = tuple(shape), int(np.prod(shape)), 4096, 4 * int(np.prod(shape))


class Api:
    def __init__(self):
        self.calls, self.fails = [], {}

    def __getattr__(self, name):
        def call(*a):
            self.calls.append(name)
            if name in self.fails:
                raise RuntimeError(self.fails[name])
        return call


@pytest.fixture
def model(monkeypatch):
    api = Api()
    monkeypatch.setattr(layered, "api", api)
    monkeypatch.setattr(paged_cache, "api", api)
    monkeypatch.setattr(layered, "leave_open", lambda: None)         # process-wide state of the current stream
    monkeypatch.setattr(layered, "GPUArray", Array)
    monkeypatch.setattr(paged_cache, "GPUArray", Array)
    monkeypatch.setattr(paged_cache, "zeros", Array)
    # an object that takes the place, and so the identity, of the one before it
    monkeypatch.setattr(layered, "RowBuffers", lambda config, rows, _one=SimpleNamespace(): vars(_one).update(rows=rows) or _one)
    m = object.__new__(layered.LayeredCausalModel)
    m.config, m.dtype, m.blocks, m.runs, m.trace_hook = SimpleNamespace(vocab_size=10), "bfloat16", [], [], None
    m.use_graphs, m._graphs, m._gstream, m._last_stream = True, layered.StepGraphs(), None, None
    m._graphs_of, m._buf, m._meta, m._out, m._ws = 0, None, None, None, None
    m._tile_sizes, m._tops = set(), set()
    m.cache = paged_cache.PagedKVCache([(1, 8, 8)], tokens_hint=1 << 18, slots=40, state_shapes=[(8,)])
    m.ran, m.captures = [], []
    m._forward = lambda ctx: m.ran.append(ctx.T)

    class Graph:
        _exec = 1

        def capture(self, stream):
            import contextlib
            m.captures.append(1)
            if "graph_end" in api.fails:
                raise RuntimeError(api.fails["graph_end"])
            return contextlib.nullcontext()

    monkeypatch.setattr(layered, "CudaGraph", Graph)
    monkeypatch.setattr(layered, "Stream", lambda: None)
    m.api = api
    return m


def decode(m, ids, times=1):
    for _ in range(times):
        m.step_device([(i, [1], [0]) for i in ids])


def start(m, ids, n=3):
    m.step_device([(i, [1] * n, [n - 1]) for i in ids])


def captured(m, ids):
    """decode steps until one is replayed; another one of the same kind then is no new capture"""
    for _ in range(40):
        if m._graphs:
            break
        decode(m, ids)
    n = len(m.captures)
    decode(m, ids)
    assert m._graphs and len(m.captures) == n


def grow_rows(m):
    m.step_device([("long", [1] * (m._buf.rows + 1), [])])


def grow_pages(m):
    ptrs = [a.device_ptr for a in m.cache.k]
    m.step_device([("much", [1] * (m.cache.pool.free_pages * 64 + 1), [])])
    assert [a.device_ptr for a in m.cache.k] == ptrs         # the fault's condition: the same address, another array


def grow_slots(m):
    start(m, [f"more{i}" for i in range(40)], 1)


@pytest.mark.parametrize("grow", [grow_rows, grow_pages, grow_slots, lambda m: m._workspace(1 << 24), lambda m: m._meta_buffer(1 << 20),
                                  lambda m: m._logits(100)], ids=["rows", "pages", "slots", "workspace", "description", "logits"])
def test_no_captured_step_outlives_an_array_of_its_launches(model, grow):
    """Addresses and identities of freed arrays come back; a captured step that names the arrays before must not."""
    m = model
    start(m, "ab")
    captured(m, "ab")
    replays = m.api.calls.count("graph_launch")
    grow(m)
    decode(m, "ab")
    assert m.api.calls.count("graph_launch") == replays      # launched one by one, on the new arrays
    captured(m, "ab")


def test_captured_steps_stay_while_the_arrays_do(model):
    m = model
    start(m, "abc")
    for ids in ("abc", "ab", "a"):
        decode(m, ids, 5)
    n = len(m.captures)
    start(m, "d")
    m.release("d")
    for ids in ("abc", "ab", "a"):
        decode(m, ids)
    assert len(m.captures) == n


def churn(m, period, steps):
    """decode steps of kinds that come by turns: `period` of them, 9 to 32 requests and different key slices"""
    ids = [f"r{i}" for i in range(32)]
    start(m, ids, 1)
    m._logits(32), m._meta_buffer(1 << 16)
    m.blocks = [SimpleNamespace(mixer=SimpleNamespace(key_slices=lambda ctx: m.plan))]
    m.plan = 0
    for i in range(steps):
        m.plan, n = divmod(i % period, 24)
        decode(m, ids[:9 + n])


@pytest.mark.parametrize("period", [24, 64, 65, 100, 300])
def test_steps_whose_kind_changes_are_not_captured_again_and_again(model, period):
    """What fits is captured once; what does not runs as single launches, a capture at most every sixteenth time of its kind."""
    m = model
    churn(m, period, 20 * period)
    assert len(m._graphs) == min(period, 64)
    assert len(m.captures) <= min(period, 64) + (period > 64) * 20 * period // 16


def test_kinds_that_come_no_more_make_room(model):
    m = model
    churn(m, 64, 64 * 6)
    assert len(m._graphs) == 64
    n, ids = len(m.captures), [f"r{i}" for i in range(20)]
    m.plan = 7                                               # contexts have grown
    decode(m, ids, 16)
    assert len(m.captures) == n + 1 and len(m._graphs) == 64
    decode(m, ids, 50)
    m.plan = 0
    decode(m, ids)                                           # used last before that: still there
    assert len(m.captures) == n + 1


@pytest.mark.parametrize("call", ["graph_end", "graph_launch"])
def test_a_step_whose_graph_finds_no_room_runs_as_single_launches(model, call):
    """The memory of a graph's own allocations is had when it is made or launched; single launches take other kernels where there is none."""
    m = model
    start(m, "ab")
    m.api.fails = {call: "cudaGraph... failed: out of memory"}
    before = len(m.ran)
    decode(m, "ab", 10)
    assert len(m.ran) - before == 10 + (call == "graph_launch") and len(m.captures) == 1 and not m._graphs     # (a capture runs the launches' code, too)
    decode(m, "a", 10)
    assert len(m.captures) == 2
    m.api.fails = {}
    grow_rows(m)
    captured(m, "ab")                                        # another try once the arrays are others
    m.api.fails = {"graph_launch": "an illegal address"}
    with pytest.raises(RuntimeError, match="illegal"):
        decode(m, "ab")
