"""rf_plan_launch's result: in the caller's device buffer, aligned for the result's fields or not, in
pinned host memory, or in none; under CUDA graph capture too.  The bits are rf_plan_run's."""
import ctypes

import pytest

from reffine_gb300 import cudart, workloads as W
from reffine_gb300.engine import from_c

pytestmark = pytest.mark.gpu


def query(eng, which):
    if which == "filter_sum":
        t = W.filter_sum_table(50_003, seed=4)
        fn = W.filter_sum_query(t.get_data_type())
    else:
        t = W.groupby_table(50_003, seed=4)
        fn = W.groupby_query(t.get_data_type())
    return eng.compile(fn), eng.upload(t)


def copied(eng, ptr, size):
    eng.sync()
    buf = (ctypes.c_ubyte * size)()
    assert cudart.rt().cudaMemcpy(buf, ctypes.c_void_p(ptr), ctypes.c_size_t(size), 4) == 0
    return buf


@pytest.mark.parametrize("which", ["filter_sum", "groupby"])
@pytest.mark.parametrize("where", ["device", "pinned"])
@pytest.mark.parametrize("offset", [0, 8, 16, 24])
def test_result_in_the_callers_buffer(eng, which, where, offset):
    plan, dt = query(eng, which)
    args, size = plan.args(dt), plan.info.output_size
    ref = plan.run(dt)
    rt, base = cudart.rt(), ctypes.c_void_p()
    if where == "device":
        assert rt.cudaMalloc(ctypes.byref(base), size + 64) == 0
        free = rt.cudaFree
    else:
        assert rt.cudaHostAlloc(ctypes.byref(base), ctypes.c_size_t(size + 64), 0) == 0
        free = rt.cudaFreeHost
    try:
        fill = (ctypes.c_ubyte * (size + 64))(*([0xA5] * (size + 64)))
        assert rt.cudaMemcpy(base, fill, ctypes.c_size_t(size + 64), 4) == 0
        plan.launch(args, 1, base.value + offset)
        raw = bytes(copied(eng, base.value, size + 64))
        assert set(raw[:offset]) <= {0xA5} and set(raw[offset + size:]) == {0xA5}  # nothing around it is touched
        out = plan.new_out()
        ctypes.memmove(ctypes.byref(out), raw[offset:offset + size], size)
        assert from_c(out) == ref
    finally:
        free(base)


def test_result_under_capture(eng):
    # a launch captured in a CUDA graph writes its result at each replay
    plan, dt = query(eng, "groupby")
    args, size = plan.args(dt), plan.info.output_size
    ref = plan.run(dt)
    rt, s = cudart.rt(), ctypes.c_void_p()
    buf = cudart.DeviceBuffer(size + 16)
    graph, exec_ = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    try:
        assert rt.cudaStreamBeginCapture(s, 1) == 0  # thread-local mode
        st = eng.lib.rf_plan_launch(plan.h, args, 1, buf.ptr.value, s)
        assert rt.cudaStreamEndCapture(s, ctypes.byref(graph)) == 0
        eng.check(st)
        assert rt.cudaGraphInstantiate(ctypes.byref(exec_), graph, ctypes.c_ulonglong(0)) == 0
        for _ in range(3):
            buf.memset(s.value, 0)
            assert rt.cudaGraphLaunch(exec_, s) == 0
            cudart.stream_sync(s.value)
            out = plan.new_out()
            ctypes.memmove(ctypes.byref(out), copied(eng, buf.ptr.value, size), size)
            assert from_c(out) == ref
    finally:
        if exec_.value:
            rt.cudaGraphExecDestroy(exec_)
        if graph.value:
            rt.cudaGraphDestroy(graph)
        rt.cudaStreamDestroy(s)
