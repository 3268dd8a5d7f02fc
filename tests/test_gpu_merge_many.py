"""Inner merges of three and four vectors at the edges of the merge kernels' tiles: windows larger than the
buffer in shared memory, runs of one key across tiles, sides of a tile and one row more - against the oracle."""
import numpy as np
import pytest

from oracle import loopgen
from parity import assert_table_same
from reffine_gb300.ir import _add, _func, _get, _in, _op, _sym, _i64_t
from test_gpu_materialize import plan_run_table
from test_gpu_tiles import key_table, spread

pytestmark = pytest.mark.gpu

SIDES = {
    "tile": [np.arange(2048), np.arange(0, 4096, 2), np.arange(2049)],
    "runs": [[0] + [7] * 5000 + [9] * 3, [0] + [7] * 4500 + [8] * 2100 + [9], [0, 1] + [7] * 4600 + [9]],
    "windows": [[0, 40_000, 40_001, 99_999], spread(60_000, 100_000, 1), spread(30_000, 100_000, 2)],
    "four": [spread(5000, 4000, 3), spread(9000, 4000, 4), spread(2049, 4000, 5), spread(20_000, 4000, 6)],
    "one": [[0], [0], [0], [0]],
}


@pytest.mark.parametrize("vectorize", [False, True])
@pytest.mark.parametrize("name", list(SIDES))
def test_merges_of_many_vectors(eng, name, vectorize):
    tabs = [key_table(k, i) for i, k in enumerate(SIDES[name])]
    t = _sym("t", _i64_t)
    vecs = [_sym("v%d" % i, tab.get_data_type()) for i, tab in enumerate(tabs)]
    space, total = _in(t, vecs[0]), _get(vecs[0][t], 0)
    for v in vecs[1:]:
        space, total = space & _in(t, v), _add(total, _get(v[t], 0))
    op = _op([t], space, [total] + [_get(v[t], 0) for v in vecs])
    os_ = _sym("op", op)
    fn = _func("merge", os_, vecs)
    fn.tbl[os_] = op
    plan = eng.compile(fn, vectorize)
    assert plan.kind == 6
    out = plan_run_table(eng, plan, *tabs)
    ref = loopgen.Query(fn, vectorize)(*tabs)
    if not vectorize:
        assert_table_same(out, ref)
        return
    v = np.ones(out["len"], bool) if out["valid"][0] is None else out["valid"][0]
    w = np.ones(ref["len"], bool) if ref["valid"] is None else ref["valid"]
    for g, r in zip(out["cols"], ref["cols"]):
        np.testing.assert_array_equal(g[v], r[w])
