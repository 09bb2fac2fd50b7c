"""Bounded waits: one that runs out ends its kernel, and the next call that synchronises says so -- once."""
import ctypes as C
import time

import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200 import llm
from pygpukit_b200._lib import api
from pygpukit_b200.core.stream import Stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sync", ["device", "stream", "read"])
def test_a_wait_that_runs_out_is_reported(sync):
    out = gk.from_numpy(np.full(1, 7, np.int32))
    api.wait_probe(1, out.device_ptr, None)              # loads the kernel
    with pytest.raises(RuntimeError, match="ran out"):
        api.device_sync()
    st = Stream()
    t = time.perf_counter()
    api.wait_probe(2000, out.device_ptr, st.handle)
    with pytest.raises(RuntimeError, match="wait_probe failed: a wait inside its kernel ran out"):
        if sync == "device":
            api.device_sync()
        elif sync == "stream":
            st.synchronize()
        else:
            out.to_numpy()
            api.device_sync()
    assert 2e-3 <= time.perf_counter() - t < 1.0         # the limit, and not much more
    api.device_sync()                                    # reported once
    assert out.to_numpy()[0] == 0
    a, w = gk.from_numpy(np.ones((40, 128), np.float32)), gk.from_numpy(np.full((64, 128), 0x3F80, np.uint16))
    c = gk.zeros((40, 64), gk.float32)
    llm.LinearRows(w).forward(a.device_ptr, 128, 40, c.device_ptr, 64)       # the device is as usable as before
    assert (c.to_numpy() == 128).all()
    for query in (api.gemm_rows_wait_error, api.gemm_fp8_wait_error, api.seq_attention_wait_error):
        err = C.c_int(7)
        query(C.byref(err))
        assert err.value == 0


@pytest.mark.parametrize("limit", [0, -1, 100001])
def test_the_limit_of_the_probe_is_bounded(limit):
    out = gk.from_numpy(np.full(1, 7, np.int32))
    with pytest.raises(RuntimeError, match="limit"):
        api.wait_probe(limit, out.device_ptr, None)
    assert out.to_numpy()[0] == 7
