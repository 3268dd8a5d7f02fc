"""Edges of the tiles of the table-result kernels: sizes around a tile and a word, nothing and
everything passing, ranges that start inside a word - against the oracle."""
import numpy as np
import pytest

from oracle import loopgen
from parity import assert_same, assert_table_same
from reffine_gb300.ir import _add, _f64, _func, _get, _gt, _i64, _in, _lt, _new, _op, _red, _sym, _i64_t
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


def key_table(keys, seed=0):
    keys = np.asarray(keys, dtype=np.int64)
    v = np.random.default_rng(seed + len(keys)).integers(-1000, 1000, len(keys))
    return Table.from_arrays(1, {"k": keys, "v": v})


def spread(n, hi, seed):
    k = np.sort(np.random.default_rng(seed).integers(0, hi, n))
    k[0] = 0
    return k


MERGES = {  # left, right: long runs of one key across tiles, windows larger than the buffer, sides that end first
    "equal_runs": ([0] + [7] * 5000 + [9] * 3, [0] + [7] * 4500 + [8] * 2100 + [9]),
    "sparse_left": ([0, 40_000, 40_001, 99_999], spread(60_000, 100_000, 1)),
    "sparse_right": (spread(60_000, 100_000, 2), [0, 1, 50_000, 99_999, 99_999]),
    "tile": (np.arange(2048), np.arange(0, 4096, 2)), "tile_plus": (np.arange(2049) // 2, np.arange(4097) // 3),
    "ends_first": (spread(5000, 1000, 3), spread(5000, 30_000, 4)), "one": ([0], [0]),
    "clusters": (np.repeat(np.arange(0, 60_000, 3000), 700), np.concatenate([[0], np.arange(1, 50_000), [57_000] * 5000])),
}


@pytest.mark.parametrize("vectorize", [False, True])
@pytest.mark.parametrize("mode", ["inner", "outer"])
@pytest.mark.parametrize("name", list(MERGES))
def test_merges_at_tile_edges(eng, name, mode, vectorize):
    a, b = (key_table(k, i) for i, k in enumerate(MERGES[name]))
    t, left, right = _sym("t", _i64_t), _sym("left", a.get_data_type()), _sym("right", b.get_data_type())
    space = _in(t, left) & _in(t, right) if mode == "inner" else _in(t, left) | _in(t, right)
    op = _op([t], space, [_get(left[t], 0), _get(right[t], 0)])
    os_ = _sym("op", op)
    fn = _func("merge", os_, [left, right])
    fn.tbl[os_] = op
    out = plan_run_table(eng, eng.compile(fn, vectorize), a, b)
    ref = loopgen.Query(fn, vectorize)(a, b)
    if mode == "inner" and vectorize:  # the plan emits the left side's rows, null where they pair with none
        v = np.ones(out["len"], bool) if out["valid"][0] is None else out["valid"][0]
        w = np.ones(ref["len"], bool) if ref["valid"] is None else ref["valid"]
        for g, r in zip(out["cols"], ref["cols"]):
            np.testing.assert_array_equal(g[v], r[w])
    else:
        assert_table_same(out, ref)


@pytest.mark.parametrize("ncol", [1, 2, 3, 5])
@pytest.mark.parametrize("zeros", [0.0, 0.1, 1.0])
def test_grouped_sums_with_zeros_at_tile_edges(eng, zeros, ncol):
    # one to five double-float sums (alone and in pairs); zero addends leave the fast path, one
    # negative addend at the end turns a thread's slots into doubles
    from widequery import wide_groupby_query, wide_table
    for n in (1, 511, 4095, 4096, 4097, 70_001):
        for negative in (False, True):
            t = wide_table(n, ncol, seed=n)
            rng = np.random.default_rng(n + ncol)
            for c in t.columns[3:]:
                c.data[rng.random(n) < zeros] = 0.0
                if negative:
                    c.data[-1] = -1.5
            fn = wide_groupby_query(t.get_data_type(), ncol)
            got = eng.compile(fn).run(eng.upload(t))
            assert_same(got, loopgen.Query(fn)(t))


@pytest.mark.parametrize("nsum", [0, 1, 2, 3, 4, 5, 6, 9, 12])
@pytest.mark.parametrize("n,nkeys", [(1, 1), (700, 460), (5000, 4999), (70_001, 30_000)])
def test_hash_group_by_slots(eng, n, nkeys, nsum):
    # every width of a slot's accumulators; keys that overflow their sector of four, and the key that
    # marks an empty slot.  Whole-number values: sums are exact
    rng = np.random.default_rng(n + nsum)
    keys = rng.integers(-2**62, 2**62, nkeys)
    keys[-1] = np.iinfo(np.int64).min
    cols = {"key": keys[rng.integers(0, nkeys, n)]}
    for i in range(nsum):
        cols["v%d" % i] = rng.integers(-1000, 1000, n).astype(np.float64)
    if nsum == 0:
        cols["v"] = np.zeros(n)
    t = Table.from_arrays(2, cols, name="slots")
    vec, k = _sym("vec", t.get_data_type()), _sym("k", _i64_t)
    red = _red(vec[k], lambda: _new([_f64(0)] * nsum + [_i64(0)]),
               lambda s, v: _new([_add(_get(s, i), _get(v, i)) for i in range(nsum)] + [_add(_get(s, nsum), _i64(1))]))
    rs = _sym("agg", red)
    op = _op([k], _in(k, vec), [_get(rs, i) for i in range(nsum + 1)])
    os_ = _sym("op", op)
    fn = _func("slots", os_, [vec])
    fn.tbl[rs], fn.tbl[os_] = red, op
    plan = eng.compile(fn)
    assert plan.kind == 5
    out = plan_run_table(eng, plan, t)
    order = np.argsort(out["cols"][0], kind="stable")
    uk, inv = np.unique(cols["key"], return_inverse=True)
    np.testing.assert_array_equal(out["cols"][0][order], uk)
    for i in range(nsum):
        np.testing.assert_array_equal(out["cols"][1 + i][order], np.bincount(inv, weights=cols["v%d" % i], minlength=len(uk)))
    np.testing.assert_array_equal(out["cols"][1 + nsum][order], np.bincount(inv, minlength=len(uk)))


def test_batch_of_growing_sizes_matches_alone(eng):
    # one batch reused for lists and results that grow and shrink: its buffers move under the graphs
    # kept for earlier sizes
    import ctypes
    from reffine_gb300 import workloads as W
    from reffine_gb300.engine import Batch
    t = W.filter_sum_table(5000, seed=5)
    dt = eng.upload(t)
    plans = [eng.compile(W.filter_sum_query(t.get_data_type(), day_lo=i, day_hi=900 + i)) for i in range(7)]
    alone = [p.run(dt) for p in plans]
    batch = Batch(eng, 512)
    for n in (1, 2, 1, 3, 5, 9, 2, 20, 60, 1, 150, 5, 400, 2, 400, 1):
        for i in range(n):
            batch.add(plans[i % 7], dt)
        batch.launch()
        assert batch.wait() == [alone[i % 7] for i in range(n)]
        batch.reset()
    batch.free()
