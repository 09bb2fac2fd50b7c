"""Dropped arrays: given back to the device, whoever asks for its memory, and never under a kernel that still reads the block."""
import ctypes as C
import threading

import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200._lib import api
from pygpukit_b200.core.stream import CudaGraph, Stream, use_stream

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    f, t = C.c_size_t(), C.c_size_t()
    api.mem_info(C.byref(f), C.byref(t))
    return f.value


def test_dropped_arrays_go_back_when_memory_is_asked_for():
    before = _free()
    keep = [gk.empty((8 * MB,), gk.uint8) for _ in range(40)]
    assert before - _free() >= 300 * MB
    del keep
    assert before - _free() <= 4 * MB
    for _ in range(2000):
        gk.empty((64,), gk.uint8)
    assert before - _free() <= 4 * MB


def test_a_block_is_not_used_again_while_a_stream_reads_it():
    """arrays dropped right behind the launch that reads them, on another stream, and new ones filled at once"""
    n, st = 1 << 20, Stream()
    outs = []
    for i in range(64):
        a, b = gk.from_numpy(np.full(n, i, np.float32)), gk.empty((n,), gk.float32)
        with use_stream(st):
            for _ in range(4):
                api.memcpy_d2d(b.device_ptr, a.device_ptr, 4 * n, st.handle)
        del a
        gk.from_numpy(np.full(n, -1.0, np.float32))
        outs.append(b)
    st.synchronize()
    assert all((b.to_numpy() == i).all() for i, b in enumerate(outs))


def test_threads_drop_arrays_at_the_same_time():
    before = _free()

    def work():
        for i in range(300):
            gk.empty((1 + 4096 * (i % 7),), gk.uint8)

    ts = [threading.Thread(target=work) for _ in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert before - _free() <= 4 * MB


def test_a_dropped_array_is_free_for_other_allocators_at_once():
    """asked of the driver, as another library of the process would find it"""
    def free():
        f, t = C.c_size_t(), C.c_size_t()
        assert C.CDLL("libcuda.so.1").cuMemGetInfo_v2(C.byref(f), C.byref(t)) == 0
        return f.value

    gk.empty((1,), gk.uint8)
    before = free()
    for _ in range(4):
        a = gk.empty((8 * MB,), gk.uint8)
        assert before - free() >= 8 * MB
        del a
        assert before - free() <= 4 * MB


def test_asking_for_the_memory_inside_a_capture():
    a, b = gk.from_numpy(np.arange(64, dtype=np.float32)), gk.empty((64,), gk.float32)
    for i in range(8):
        gk.empty((64,), gk.uint8)
    g, st = CudaGraph(), Stream()
    with g.capture(st):
        assert _free() > 0
        api.memcpy_d2d(b.device_ptr, a.device_ptr, 256, st.handle)
    g.replay()
    st.synchronize()
    assert np.array_equal(b.to_numpy(), np.arange(64, dtype=np.float32))
