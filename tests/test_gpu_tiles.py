"""Edges of the tiles of the table-result kernels: sizes around a tile and a word, nothing and
everything passing, ranges that start inside a word - against the oracle."""
import numpy as np
import pytest

from oracle import loopgen
from parity import assert_table_same
from reffine_gb300.ir import _add, _func, _get, _gt, _i64, _in, _lt, _op, _sym, _i64_t
from reffine_gb300.table import Table
from test_gpu_materialize import plan_run_table

pytestmark = pytest.mark.gpu


def filtered_op(t, limit, after=None):
    tt, vec = _sym("t", _i64_t), _sym("vec", t.get_data_type())
    e = vec[tt]
    f = _lt(_get(e, 0), _i64(limit))
    fs = _sym("f", f)
    space = _in(tt, vec) & fs if after is None else _in(tt, vec) & _gt(tt, _i64(after)) & fs
    op = _op([tt], space, [_add(_get(e, 0), _i64(1)), _get(e, 1)])
    os_ = _sym("op", op)
    fn = _func("flt", os_, [vec])
    fn.tbl[fs] = f
    fn.tbl[os_] = op
    return fn


@pytest.mark.parametrize("vectorize", [False, True])
@pytest.mark.parametrize("n,after", [(1, None), (31, None), (33, 0), (2047, None), (2048, 5), (2049, 31), (4097, 2046),
                                     (65_537, 32), (614_405, 40_000)])
def test_compaction_at_tile_edges(eng, vectorize, n, after):
    rng = np.random.default_rng(n)
    t = Table.from_arrays(1, {"k": np.arange(n, dtype=np.int64), "x": rng.integers(0, 100, n), "y": rng.standard_normal(n)})
    for limit in (0, 1, 37, 100):
        fn = filtered_op(t, limit, after)
        out = plan_run_table(eng, eng.compile(fn, vectorize), t)
        ref = loopgen.Query(fn, vectorize)(t)
        if not vectorize:
            assert_table_same(out, ref)
            continue
        assert out["len"] == ref["len"]
        v = np.ones(out["len"], bool) if ref["valid"] is None else ref["valid"]
        got = np.ones(out["len"], bool) if out["valid"][0] is None else out["valid"][0]
        np.testing.assert_array_equal(got, v)
        for g, r in zip(out["cols"], ref["cols"]):
            np.testing.assert_array_equal(g[v], r[v])
