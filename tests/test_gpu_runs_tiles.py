"""Edges of the tiles of the run-end segmented reduce: runs that end at, before and after a thread's
and a tile's last item, runs longer than many tiles, empty runs - against the oracle."""
import numpy as np
import pytest

from oracle import loopgen
from parity import assert_table_same
from reffine_gb300 import ir
from reffine_gb300.ir import _add, _func, _get, _gt, _i64, _in, _max, _new, _op, _red, _sel, _sym, _i64_t, _f64
from reffine_gb300.table import Table
from test_gpu_materialize import plan_run_table

pytestmark = pytest.mark.gpu

TILE = 256 * 11  # items of a tile that stages one double a row


def grouped_query(tbl_type, wide):
    vec, t = _sym("vec", tbl_type), _sym("t", _i64_t)
    if wide:  # four columns staged: a smaller tile, conditional and idempotent leaves
        red = _red(vec[t], lambda: _new([_f64(0), _i64(0), _i64(-5000), _i64(0)]),
                   lambda s, v: _new([_add(_get(s, 0), _get(v, 0)), _add(_get(s, 1), _i64(1)), _max(_get(s, 2), _get(v, 1)),
                                      _sel(_gt(_get(v, 1), _i64(0)), _add(_get(s, 3), _get(v, 2)), _get(s, 3))]))
        n = 4
    else:
        red = _red(vec[t], lambda: _new([_f64(0), _i64(0)]),
                   lambda s, v: _new([_add(_get(s, 0), _get(v, 0)), _add(_get(s, 1), _i64(1))]))
        n = 2
    rs = _sym("agg", red)
    op = _op([t], _in(t, vec), [_get(rs, k) for k in range(n)])
    os_ = _sym("op", op)
    fn = _func("runs", os_, [vec])
    fn.tbl[rs] = red
    fn.tbl[os_] = op
    return fn


LENGTHS = {
    "one": [1], "ones": [1] * (3 * TILE), "tile": [TILE - 1, TILE - 1, 1, TILE, TILE + 1], "thread": [10, 11, 12, 9] * 700,
    "long": [3, 20 * TILE + 5, 1, 7], "mixed": list(np.random.default_rng(3).geometric(0.05, 9000)) + [50_000, 1, 1],
    "empty_runs": [4, 0, 0, 9, 0, TILE, 0, 1],
}


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("name", list(LENGTHS))
def test_runs_at_tile_edges(eng, name, wide):
    lens = np.array(LENGTHS[name], dtype=np.int64)
    n = int(lens.sum())
    rng = np.random.default_rng(len(lens))
    cols = {"key": np.arange(len(lens), dtype=np.int64) * 5 - 7, "v": rng.uniform(0.0, 1000.0, n)}
    if wide:
        cols.update(a=rng.integers(-1000, 1000, n), b=rng.integers(-99, 99, n))
    t = Table.from_arrays(2, cols, runend={"key": lens.cumsum().astype(np.int32)})
    fn = grouped_query(t.get_data_type(), wide)
    plan = eng.compile(fn)
    assert plan.kind == 4
    out = plan_run_table(eng, plan, t)
    assert_table_same(out, loopgen.Query(fn)(t))
    np.testing.assert_array_equal(out["cols"][2], lens)
    again = plan_run_table(eng, plan, t)
    for a, b in zip(out["cols"], again["cols"]):
        np.testing.assert_array_equal(a, b)  # the tiles alone set the order of the sums
