"""Run-end segmented reduce at the edges of its own geometry: columns of no runs, and run lengths
around a thread's and a tile's items for both widths of the staged row - against the oracle."""
import numpy as np
import pytest

from oracle import loopgen
from parity import assert_table_same
from reffine_gb300.table import Table
from test_gpu_materialize import plan_run_table
from test_gpu_runs_tiles import grouped_query

pytestmark = pytest.mark.gpu


def runs_table(lens, wide, seed=0):
    lens = np.array(lens, dtype=np.int64)
    n = int(lens.sum())
    rng = np.random.default_rng(seed)
    cols = {"key": np.arange(len(lens), dtype=np.int64) * 5 - 7, "v": rng.uniform(0.0, 1000.0, n)}
    if wide:
        cols.update(a=rng.integers(-1000, 1000, n), b=rng.integers(-99, 99, n))
    return Table.from_arrays(2, cols, runend={"key": lens.cumsum().astype(np.int32)})


@pytest.mark.parametrize("vectorize", [False, True])
@pytest.mark.parametrize("wide", [False, True])
def test_no_runs(eng, wide, vectorize):
    # on a new plan, after a table of many tiles on the same plan (whose tile bounds the plan's
    # buffer then holds), and before another
    empty, full = runs_table([], wide), runs_table([3] * 20_000, wide)
    plan = eng.compile(grouped_query(empty.get_data_type(), wide), vectorize)
    assert plan.kind == 4
    ref = loopgen.Query(grouped_query(full.get_data_type(), wide), vectorize)(full)
    for t in (empty, full, empty, full):
        out = plan_run_table(eng, plan, t)
        if t is empty:
            assert out["len"] == 0 and all(len(c) == 0 for c in out["cols"])
        else:
            assert_table_same(out, ref)


def geometry(wide):
    """Items of a thread and of a tile of 128 threads: a staged row and its run end share 36 KiB."""
    row_bytes = 4 + 8 * (3 if wide else 1)
    k = max(1, min(22, 36 * 1024 // (128 * row_bytes)))
    return k, 128 * k


def lengths(shape, k, tile):
    # a run takes an item a row and one for its end
    return {"thread": [k - 2, k - 1, k, k + 1, 1] * 400,
            "tile": [tile - 2, tile - 1, tile, tile + 1, 1, tile - 1, 2 * tile - 1],
            "whole": [tile - 1] * 3, "one_over": [tile - 1] * 3 + [0], "one_short": [tile - 1] * 2 + [tile - 2],
            "one_run": [3 * tile - 1], "one_run_over": [3 * tile], "ends_only": [0] * (2 * tile) + [5]}[shape]


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("shape", ["thread", "tile", "whole", "one_over", "one_short", "one_run", "one_run_over", "ends_only"])
def test_runs_at_the_kernels_own_edges(eng, shape, wide):
    t = runs_table(lengths(shape, *geometry(wide)), wide, seed=len(shape))
    fn = grouped_query(t.get_data_type(), wide)
    out = plan_run_table(eng, eng.compile(fn), t)
    assert_table_same(out, loopgen.Query(fn)(t))
