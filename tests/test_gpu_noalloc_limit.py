"""rf_plan_run_noalloc near the limit of its fixed scratch: a run that fits with the plan's own tiles is
not refused because a smaller tiling would run faster."""
import ctypes

import pytest

from oracle import loopgen
from parity import assert_same
from reffine_gb300 import _capi, engine, workloads as W

pytestmark = pytest.mark.gpu


def test_small_scratch_takes_fewer_units(eng, monkeypatch):
    n = 100_003  # 13 units of 8192 rows, 25 of 4096
    t = W.filter_sum_table(n, seed=3)
    fn = W.filter_sum_query(t.get_data_type())
    plan = eng.compile(fn)
    args = plan.args(eng.upload(t))
    fixed, acc = 768 + 256, 16  # counter, loop bounds and result; a unit's sum and count
    got = []
    for limit in (fixed + 25 * acc, fixed + 13 * acc, fixed + 12 * acc):
        monkeypatch.setenv("RF_NOALLOC_LIMIT", str(limit))
        out = plan.new_out()
        st = eng.lib.rf_plan_run_noalloc(plan.h, args, 1, ctypes.byref(out), None)
        got.append(st)
        if st == _capi.RF_OK:
            assert_same(engine.from_c(out), loopgen.Query(fn)(t))
    assert got == [_capi.RF_OK, _capi.RF_OK, _capi.RF_ERR_INVALID]
