"""Device memory of table-result plans: what grows with the inputs goes back to the pool when a run
ends, and a server counts it before it admits the run."""
import ctypes

import numpy as np
import pytest

from reffine_gb300 import engine as E, serve, workloads as W
from reffine_gb300.ir import _func, _get, _in, _op, _sym, _i64_t
from reffine_gb300.table import Table
from test_gpu_tiles import filtered_op
from test_zz_no_alloc import _device_memory

pytestmark = pytest.mark.gpu

N = 600_000


def merge(mode):
    a, b = (Table.from_arrays(1, {"k": np.arange(N, dtype=np.int64) * s, "v": np.arange(N, dtype=np.int64)}) for s in (2, 3))
    t, left, right = _sym("t", _i64_t), _sym("left", a.get_data_type()), _sym("right", b.get_data_type())
    space = _in(t, left) & _in(t, right) if mode == "inner" else _in(t, left) | _in(t, right)
    op = _op([t], space, [_get(left[t], 0), _get(right[t], 0)])
    os_ = _sym("op", op)
    fn = _func("merge", os_, [left, right])
    fn.tbl[os_] = op
    return fn, [a, b]


def case(which):
    """A query, its tables and the bytes of its scratch that grow with them, at the least."""
    if which == "select":
        t = Table.from_arrays(1, {"k": np.arange(40 * N, dtype=np.int64), "x": np.arange(40 * N) % 100, "y": np.zeros(40 * N)})
        return filtered_op(t, 37), [t], 5 * N  # a bit an element
    if which == "runs":
        t = Table.from_arrays(2, {"key": np.arange(N, dtype=np.int64), "value": np.ones(2 * N)},
                              runend={"key": (2 * np.arange(1, N + 1)).astype(np.int32)})
        return W.hashgroup_query(t.get_data_type()), [t], 16 * N  # a state a run
    fn, tabs = merge(which)
    return fn, tabs, 8 * N  # a partner a row


def run(eng, plan, args, n):
    h = ctypes.c_void_p()
    eng.check(eng.lib.rf_plan_run(plan.h, args, n, ctypes.byref(h), None))
    out = E.DeviceTable(eng, h, plan.fn.output.type, [])
    rows = out.export()["len"]
    out.free()
    return rows


@pytest.mark.parametrize("which", ["select", "runs", "inner", "outer"])
def test_scratch_goes_back_when_a_run_ends(eng, which):
    fn, tabs, scratch = case(which)
    dts = [eng.upload(t, None, True) for t in tabs]
    plans = [eng.compile(fn) for _ in range(4)]
    eng.sync()
    before = _device_memory()[2]
    rows = [run(eng, p, p.args(*dts), len(dts)) for p in plans for _ in range(2)]
    eng.sync()
    assert len(set(rows)) == 1 and rows[0] > 0
    assert _device_memory()[2] - before < scratch  # the four plans together hold less than one's


@pytest.mark.parametrize("which", ["select", "runs", "inner", "outer"])
def test_a_server_counts_the_scratch(eng, which):
    fn, tabs, scratch = case(which)
    dts = [eng.upload(t, None, True) for t in tabs]
    plan = eng.compile(fn)
    eng.sync()
    srv = serve.Server(eng, "per_query")
    out = srv.submit(plan, *dts, tag=1)
    for _ in range(200):
        if srv.poll(4, 50_000):
            break
    peak = srv.stats()["peak_inflight_bytes"]
    srv.close()
    E.DeviceTable(eng, out, fn.output.type, []).free()
    elements = {"select": 40 * N, "runs": N, "inner": N, "outer": 2 * N}[which]
    assert peak >= elements * (8 + 8 * len(fn.output.type.dtypes)) + scratch
