"""The work this backend is timed on: compiled queries over device-resident tables, called as a
program calls them (Engine.compile / Plan.run / Plan.launch / rf_plan_run / rf_batch_*).

A case names a query shape of reffine_gb300.workloads or of the reference's own tests, the sizes
of its tables and the options of the call.  Inputs are made on the GPU from the seed alone with
the value distributions of reffine_gb300.workloads, copied to pinned host memory as Arrow columns
and uploaded with Engine.upload, which is how a table reaches the device; the plan is compiled
and the index of a probed or walked table built beforehand, as a program does once per table.
"""
import ctypes
import math

import numpy as np
import torch

from reffine_gb300 import ir
from reffine_gb300 import workloads as W
from reffine_gb300.engine import DeviceTable, Engine, compile_op
from reffine_gb300.table import Table

KINDS = ("filter_sum", "groupby", "hashgroup", "join", "runs", "select", "merge", "batch")


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # one small query and its answer: the latency of a call (the serving mix holds tables from
        # a thousand rows up)
        {"name": "filter_sum_10k", "kind": "filter_sum", "rows": 10_007, "nulls": 0.0, "call": "run"},
        # the filter + sum benchmark table
        {"name": "filter_sum_6M", "kind": "filter_sum", "rows": 6_000_000, "nulls": 0.0, "call": "run"},
        # a mid-size group-by enqueued without waiting, its answer left on the device
        {"name": "groupby_1M_launch", "kind": "groupby", "rows": 1_000_003, "nulls": 0.0, "call": "launch"},
        # the low-cardinality group-by benchmark table
        {"name": "groupby_60M", "kind": "groupby", "rows": 60_000_000, "nulls": 0.0, "call": "run"},
        # high-cardinality group-by over unsorted skewed keys: a mid-size table, and the benchmark's
        {"name": "hashgroup_1M", "kind": "hashgroup", "rows": 1_000_003, "keys": 100_000, "skew": 1.1, "nulls": 0.0},
        {"name": "hashgroup_100M", "kind": "hashgroup", "rows": 100_000_000, "keys": 10_000_000, "skew": 1.1,
         "nulls": 0.0},
        # the filtered join + aggregate benchmark tables
        {"name": "join_10M_200M", "kind": "join", "build": 10_000_000, "rows": 200_000_000, "call": "run"},
        # the reference's own grouped form: rows sorted by key, the key run-end encoded
        {"name": "runs_20M", "kind": "runs", "rows": 20_000_003, "keys": 2_000_000, "skew": 1.1},
        # an Op that keeps the rows passing a filter in a new table
        {"name": "select_20M", "kind": "select", "rows": 20_000_003, "percent": 37, "vectorize": False},
        # merge co-iteration of two sorted tables: both sides hold the key, or either does
        {"name": "merge_inner_5M", "kind": "merge", "mode": "inner", "left": 5_000_011, "right": 4_000_037,
         "overlap": 0.6, "value": "i64"},
        {"name": "merge_outer_3M", "kind": "merge", "mode": "outer", "left": 3_000_017, "right": 2_500_009,
         "overlap": 0.4, "value": "f64"},
        # a mix of small queries of three shapes with constants of their own, in one batch
        {"name": "batch_64", "kind": "batch", "queries": 64, "rows": 1_000_003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(KINDS)
    if kind == "filter_sum":
        c = {"rows": _log(rng, 1_000, 50_000_000), "nulls": rng.choice([0.0, 0.05]), "call": rng.choice(["run", "launch", "host"])}
        if c["call"] == "host":  # the drop-in call copies its host table each time
            c["rows"] = min(c["rows"], 6_000_000 + rng.randrange(64))
    elif kind == "groupby":
        c = {"rows": _log(rng, 1_000, 60_000_000), "nulls": rng.choice([0.0, 0.05]), "call": rng.choice(["run", "launch"])}
    elif kind == "hashgroup":
        rows = _log(rng, 1_000, 100_000_000)
        c = {"rows": rows, "keys": max(1, min(10_000_000, int(rows * math.exp(rng.uniform(math.log(1e-3), math.log(0.5)))))),
             "skew": rng.choice([0.0, 1.1]), "nulls": rng.choice([0.0, 0.05])}
    elif kind == "join":
        c = {"build": _log(rng, 1_000, 10_000_000), "rows": _log(rng, 10_000, 200_000_000), "call": rng.choice(["run", "launch"])}
    elif kind == "runs":
        rows = _log(rng, 1_000, 20_000_003)
        c = {"rows": rows, "keys": max(1, int(rows / math.exp(rng.uniform(math.log(2), math.log(1000))))),
             "skew": rng.choice([0.0, 1.1])}
    elif kind == "select":
        c = {"rows": _log(rng, 1_000, 20_000_003), "percent": rng.randint(1, 99), "vectorize": rng.random() < 0.5}
    elif kind == "merge":
        c = {"mode": rng.choice(["inner", "outer"]), "left": _log(rng, 1_000, 5_000_011), "right": _log(rng, 1_000, 5_000_011),
             "overlap": rng.choice([0.1, 0.5, 0.95]), "value": rng.choice(["i64", "f64"])}
    else:
        c = {"queries": rng.randint(4, 64), "rows": _log(rng, 10_000, 2_000_000)}
    return {"kind": kind, **c}


# ----------------------------------------------------------------------------- columns, on the GPU
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _ints(g, n, lo, hi, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=dtype)


def _filter_sum_cols(g, n):
    return {"day": _ints(g, n, 0, 2557, torch.int32), "price": _uniform(g, n, 900.0, 105000.0),
            "discount": _ints(g, n, 0, 11).double() / 100.0, "quantity": _ints(g, n, 1, 51).double()}


def _groupby_cols(g, n):
    return {"flag_a": _ints(g, n, 0, 3, torch.int8), "flag_b": _ints(g, n, 0, 2, torch.int8),
            "qty": _ints(g, n, 1, 51).double(), "price": _uniform(g, n, 900.0, 105000.0), "disc": _uniform(g, n, 0.0, 0.1),
            "tax": _uniform(g, n, 0.0, 0.08), "day": _ints(g, n, 0, 2557, torch.int32)}


def _ranks(g, n, nkeys, skew):
    """n ranks in [0, nkeys): Zipf(skew) by inverse CDF, or uniform."""
    if not skew:
        return _ints(g, n, 0, nkeys)
    # in whole numbers, whose running sum has the same bits each time
    cdf = (torch.arange(1, nkeys + 1, device="cuda", dtype=torch.float64).pow_(-skew) * 2.0 ** 40).long().clamp_(min=1).cumsum_(0)
    return torch.searchsorted(cdf, _ints(g, n, 0, int(cdf[-1])), right=True)


ID_MASK = (1 << 40) - 1


def _mult(g):
    """An odd multiplier: it permutes the 2^40 ids, so distinct ranks have distinct ids."""
    return 2 * int(torch.randint(1, 1 << 38, (1,), generator=g, device="cuda")) + 1


def _hash_cols(g, case):
    """The columns, and the multiplier that made the keys of their ranks."""
    mult = _mult(g)
    key = (_ranks(g, case["rows"], case["keys"], case["skew"]) * mult) & ID_MASK
    return {"key": key, "value": _uniform(g, case["rows"], 0.0, 1000.0)}, mult


def _run_cols(g, case):
    """The run values and run ends of the sorted keys, and the rows' values; every key has a row."""
    ranks = _ranks(g, case["rows"] - case["keys"], case["keys"], case["skew"])
    counts = torch.bincount(ranks, minlength=case["keys"]) + 1
    keys, order = ((torch.arange(case["keys"], device="cuda") * _mult(g)) & ID_MASK).sort()
    counts = counts[order]
    return keys, counts.cumsum(0).to(torch.int32), counts, _uniform(g, case["rows"], 0.0, 1000.0)


def _join_cols(g, nbuild, nprobe):
    keys = (torch.arange(nbuild, device="cuda") * _mult(g)) & ID_MASK
    build = {"key": keys, "attr": _ints(g, nbuild, 0, 25, torch.int32)}
    fk = keys[_ints(g, nprobe, 0, nbuild)]
    miss = _ints(g, nprobe, 1 << 41, (1 << 41) + (1 << 40))
    fk = torch.where(torch.rand(nprobe, generator=g, device="cuda") < 0.9, fk, miss)
    return build, {"fk": fk, "amount": _uniform(g, nprobe, 1.0, 10000.0), "day": _ints(g, nprobe, 0, 2557, torch.int32)}


def _select_cols(g, n):
    return {"k": torch.arange(n, device="cuda") * 3 + 7, "x": torch.randperm(n, generator=g, device="cuda") % 100,
            "y": torch.randn(n, generator=g, device="cuda", dtype=torch.float64)}


def _merge_shape(case):
    """Distinct keys of the left, of the right and of both, and how often each side holds the j-th of its keys."""
    nl, nr = case["left"] * 4 // 5 + 2, case["right"] * 4 // 5 + 2
    common = max(1, int(case["overlap"] * min(nl, nr)))
    return nl, nr, common, lambda j: 1 + (j % 4 == 1), lambda j: 1 + (j % 8 == 1) + (j % 8 == 6)


def _merge_cols(g, case):
    """Two sorted sides over one universe of keys; the first `common` keys of a random order are on both sides."""
    nl, nr, common, dup_l, dup_r = _merge_shape(case)
    ids = _ints(g, nl + nr - common, 1, 4).cumsum(0)
    order = torch.randperm(len(ids), generator=g, device="cuda")
    order[(order == 0).nonzero()[0, 0]] = order[0].clone()
    order[0] = 0  # the walk starts at the larger first key, which both sides have to hold
    sides = []
    for n, at, dup in ((case["left"], order[:nl], dup_l), (case["right"], torch.cat([order[:common], order[nl:]]), dup_r)):
        k = torch.repeat_interleave(ids[at], dup(torch.arange(len(at), device="cuda")))[:n].sort().values
        v = _ints(g, n, -1000, 1000)
        sides.append((k, v if case["value"] == "i64" else v.double() / 8 + _uniform(g, n, 0.0, 1.0)))
    return sides


def _mask(g, n, share):
    """Which rows are valid (column 1 of the table), or None where none is null."""
    return torch.rand(n, generator=g, device="cuda") >= share if share else None


# ----------------------------------------------------------------------------- tables and plans
_ENGINE = []


def _engine():
    if not _ENGINE:
        _ENGINE.append(Engine(0))
    return _ENGINE[0]


def _host(x):
    h = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    h.copy_(x)
    return h.numpy()


def _iter_col(n):
    return np.empty(n, dtype=np.int64)  # an iterator column that no query of the table reads: not uploaded


def _upload(tab, cols=None, index=False):
    dt = _engine().upload(tab, cols, index)
    _engine().sync()
    return dt


def _flat(dim, cols, n, mask=None, lead=None):
    """A host table of the GPU columns `cols`, behind an iterator column `lead` of its own if given."""
    arrays = {lead: _iter_col(n)} if lead else {}
    arrays.update((k, _host(v)) for k, v in cols.items())
    valid = None
    if mask is not None:
        valid = {list(arrays)[1]: mask.cpu().numpy()}
    return Table.from_arrays(dim, arrays, valid=valid)


def _select_query(ttype, percent):
    """The key and two outputs of the rows whose x is below `percent` (an Op over a vector, with a filter)."""
    t, vec = ir._sym("t", ir._i64_t), ir._sym("vec", ttype)
    e = vec[t]
    f = ir._lt(ir._get(e, 0), ir._i64(percent))
    f_sym = ir._sym("f", f)
    op = ir._op([t], ir._in(t, vec) & f_sym, [ir._add(ir._get(e, 0), ir._i64(1)), ir._get(e, 1)])
    op_sym = ir._sym("op", op)
    fn = ir._func("select", op_sym, [vec])
    fn.tbl[f_sym] = f
    fn.tbl[op_sym] = op
    return fn


def _merge_query(ltype, rtype, mode):
    t, left, right = ir._sym("t", ir._i64_t), ir._sym("left", ltype), ir._sym("right", rtype)
    lval, rval = ir._get(left[t], 0), ir._get(right[t], 0)
    if mode == "inner":
        op = ir._op([t], ir._in(t, left) & ir._in(t, right), [ir._add(lval, rval)])
    else:
        op = ir._op([t], ir._in(t, left) | ir._in(t, right), [ir._sub(lval, rval), lval, rval])
    op_sym = ir._sym("op", op)
    fn = ir._func("merge", op_sym, [left, right])
    fn.tbl[op_sym] = op
    return fn


def _value_state(case, fn, inputs):
    """The plan of a Reduce query and what its call needs."""
    plan = _engine().compile(fn)
    state = {"case": case, "plan": plan, "inputs": inputs}
    if case["call"] == "launch":
        state["args"] = plan.args(*inputs)
        state["out"] = torch.zeros(plan.info.output_size, dtype=torch.uint8, device="cuda")
    return state


def _batch_shapes(case):
    """(shape, rows) of the resident tables a batch reads: three shapes, three sizes each."""
    top = case["rows"]
    return [(s, max(1000, n)) for n in (top, top // 7, top // 61) for s in ("filter_sum", "groupby", "join")]


def _batch_constants(case):
    """Per query: its table and the constants of its filter."""
    got = []
    for i in range(case["queries"]):
        k = i % 9
        s = _batch_shapes(case)[k][0]
        c = {"filter_sum": {"day_lo": 100 + 7 * i, "day_hi": 700 + 23 * i}, "groupby": {"day_max": 2500 - 19 * i},
             "join": {"day_lo": 5 * i, "day_hi": 365 + 29 * i}}[s]
        got.append((k, s, c))
    return got


def prepare(case, seed):
    kind, g, eng = case["kind"], _gen(seed), _engine()
    n = case.get("rows", 0)
    if kind == "filter_sum":
        cols = _filter_sum_cols(g, n)
        tab = _flat(2, cols, n, _mask(g, n, case["nulls"]), "key")
        fn = W.filter_sum_query(tab.get_data_type())
        if case["call"] == "host":
            return {"case": case, "fn": compile_op(fn, engine=eng), "table": tab}
        return _value_state(case, fn, (_upload(tab, range(1, 5)),))
    if kind == "groupby":
        cols = _groupby_cols(g, n)
        tab = _flat(2, cols, n, _mask(g, n, case["nulls"]), "key")
        return _value_state(case, W.groupby_query(tab.get_data_type()), (_upload(tab, range(1, 8)),))
    if kind == "join":
        build, probe = _join_cols(g, case["build"], n)
        bt, pt = _flat(1, build, case["build"]), _flat(2, probe, n, None, "row")
        del build, probe
        fn = W.join_query(bt.get_data_type(), pt.get_data_type())
        return _value_state(case, fn, (_upload(bt, None, True), _upload(pt, range(1, 4))))
    if kind == "batch":
        batch = ctypes.c_void_p()
        eng.check(eng.lib.rf_batch_create(eng.h, case["queries"], ctypes.byref(batch)))
        state = {"case": case, "batch": batch, "queries": [], "plans": []}
        tabs = []
        for shape, rows in _batch_shapes(case):
            if shape == "join":
                build, probe = _join_cols(g, max(1000, rows // 20), rows)
                bt, pt = _flat(1, build, max(1000, rows // 20)), _flat(2, probe, rows, None, "row")
                tabs.append(((bt, pt), (_upload(bt, None, True), _upload(pt, range(1, 4)))))
            else:
                t = _flat(2, (_filter_sum_cols if shape == "filter_sum" else _groupby_cols)(g, rows), rows, None, "key")
                tabs.append(((t,), (_upload(t, range(1, len(t.columns))),)))
        query = {"filter_sum": W.filter_sum_query, "groupby": W.groupby_query, "join": W.join_query}
        for k, shape, const in _batch_constants(case):
            plan = eng.compile(query[shape](*[t.get_data_type() for t in tabs[k][0]], **const))
            out = np.zeros(plan.info.output_size // 8, dtype=np.float64)
            state["plans"].append((plan, tabs[k][1]))
            state["queries"].append((plan.h, plan.args(*tabs[k][1]), len(tabs[k][1]), out.ctypes.data, out))
        return state
    vectorize = bool(case.get("vectorize", False))
    if kind == "hashgroup":
        cols, mult = _hash_cols(g, case)
        tab = _flat(2, cols, n, _mask(g, n, case["nulls"]))
        tabs, index, fn = [tab], False, W.hashgroup_query(tab.get_data_type())
    elif kind == "runs":
        keys, ends, _, vals = _run_cols(g, case)
        tab = Table.from_arrays(2, {"key": _host(keys), "value": _host(vals)}, runend={"key": _host(ends)})
        tabs, index, fn = [tab], True, W.hashgroup_query(tab.get_data_type())
    elif kind == "select":
        tab = _flat(1, _select_cols(g, n), n)
        tabs, index, fn = [tab], True, _select_query(tab.get_data_type(), case["percent"])
    else:
        tabs = [_flat(1, {"t": k, "v": v}, len(k)) for k, v in _merge_cols(g, case)]
        index, fn = case["mode"] == "inner", _merge_query(*[t.get_data_type() for t in tabs], case["mode"])
    plan = eng.compile(fn, vectorize)
    inputs = tuple(_upload(t, None, index) for t in tabs)
    state = {"case": case, "plan": plan, "inputs": inputs, "args": plan.args(*inputs)}
    if kind == "hashgroup":
        state.update(stream=torch.cuda.ExternalStream(eng.stream), inverse=pow(mult, -1, 1 << 40))
    return state


# ----------------------------------------------------------------------------- one pass
class _Column:
    """A device column of a result table, for torch.as_tensor (which keeps this object, and so the table)."""

    def __init__(self, table, ptr, count, typestr):
        self.table = table
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr or 0, False), "version": 3}


def _column(table, col, typestr, part=0):
    ptr, count = ctypes.c_void_p(), ctypes.c_int64()
    table.eng.check(table.eng.lib.rf_table_column(table.h, col, part, ctypes.byref(ptr), ctypes.byref(count)))
    if not count.value:
        return torch.empty(0, dtype={"<i8": torch.int64, "<f8": torch.float64, "|u1": torch.uint8}[typestr], device="cuda")
    return torch.as_tensor(_Column(table, ptr.value, count.value, typestr), device="cuda")


def _struct(out, case):
    """A Reduce's answer on the device: per group the FP64 fields and the count that ends it."""
    groups = {"filter_sum": 1, "groupby": 6, "join": 5}[case["kind"]]
    words = out.view(torch.int64).reshape(groups, -1)
    return {"fields": words.view(torch.float64)[:, :-1], "count": words[:, -1]}


def run(state):
    case = state["case"]
    kind, eng = case["kind"], _engine()
    if kind == "batch":
        lib, b = eng.lib, state["batch"]
        eng.check(lib.rf_batch_reset(b))
        for plan, args, n, out, _ in state["queries"]:
            eng.check(lib.rf_batch_add(b, plan, args, n, out))
        eng.check(lib.rf_batch_launch(b, None))
        eng.check(lib.rf_batch_wait(b))
        fields, counts = [], []
        for (_, _, _, _, out), (_, shape, _) in zip(state["queries"], _batch_constants(case)):
            w = out.reshape({"filter_sum": 1, "groupby": 6, "join": 5}[shape], -1)
            fields.append(w[:, :-1].reshape(-1))
            counts.append(w[:, -1].copy().view(np.int64))
        return {"fields": np.concatenate(fields), "count": np.concatenate(counts)}
    if "fn" in state:
        return state["fn"](state["table"])
    plan = state["plan"]
    if case.get("call") == "run":
        return plan.run(*state["inputs"])
    if case.get("call") == "launch":
        plan.launch(state["args"], len(state["inputs"]), state["out"].data_ptr())
        return _struct(state["out"], case)
    h = ctypes.c_void_p()
    eng.check(eng.lib.rf_plan_run(plan.h, state["args"], len(state["inputs"]), ctypes.byref(h), None))
    table = DeviceTable(eng, h, plan.fn.output.type, [])
    value = "<f8" if case.get("value", "f64") == "f64" else "<i8"
    if kind == "select":
        got = [_column(table, 0, "<i8"), _column(table, 1, "<i8"), _column(table, 2, "<f8")]
        return got + [_column(table, 0, "|u1", 1)] if case["vectorize"] else got
    if kind == "merge":
        return [_column(table, 0, "<i8")] + [_column(table, c, value) for c in range(1, 2 if case["mode"] == "inner" else 4)]
    cols = [_column(table, 0, "<i8"), _column(table, 1, "<f8"), _column(table, 2, "<i8")]
    if kind == "runs":
        return cols
    # the groups of a hash group-by come in no order: the program puts them at the places of its ids
    # (on the stream that made them, whose order also keeps the table until they are read)
    with torch.cuda.stream(state["stream"]):
        at = (cols[0] * state["inverse"]) & ID_MASK
        return [torch.zeros(case["keys"], dtype=c.dtype, device="cuda").index_copy_(0, at, c) for c in cols]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _distinct(rows, nkeys, skew):
    """Expected distinct keys among `rows` draws."""
    if not skew:
        return nkeys * -math.expm1(rows * math.log1p(-1.0 / nkeys)) if nkeys > 1 else 1.0
    p = np.arange(1, nkeys + 1, dtype=np.float64) ** (-skew)
    p /= p.sum()
    return float(-np.expm1(rows * np.log1p(-np.minimum(p, 0.999999))).sum())


def _value_bytes(kind, rows, build=0, nulls=0.0):
    per = {"filter_sum": 28, "groupby": 38, "join": 20}[kind]
    return rows * per + build * 12 + (rows / 8 if nulls else 0) + {"filter_sum": 16, "groupby": 384, "join": 80}[kind]


def work(case):
    kind, n = case["kind"], case.get("rows", 0)
    if kind in ("filter_sum", "groupby", "join"):
        b = _value_bytes(kind, n, case.get("build", 0), case.get("nulls", 0.0))
    elif kind == "batch":
        b = 0
        for k, shape, _ in _batch_constants(case):
            rows = _batch_shapes(case)[k][1]
            b += _value_bytes(shape, rows, max(1000, rows // 20) if shape == "join" else 0)
    elif kind == "hashgroup":
        b = 16 * n + 24 * _distinct(n, case["keys"], case["skew"])
    elif kind == "runs":
        b = 8 * n + (12 + 24) * case["keys"]
    elif kind == "select":
        b = 24 * n + (24 * n if case["vectorize"] else 24 * n * case["percent"] / 100)
    else:
        # visits of a key: the fewer of its rows on the two sides, or the more of them
        nl, nr, common, dup_l, dup_r = _merge_shape(case)
        j = np.arange(common)
        both = int(np.minimum(dup_l(j), dup_r(j)).sum())
        b = 16 * (case["left"] + case["right"]) + (16 * both if case["mode"] == "inner" else 32 * (case["left"] + case["right"] - both))
    return {"bytes": float(b), "flops": 0.0}


# ----------------------------------------------------------------------------- the answers in 64 bits
def _filter_sum_exact(c, mask, day_lo=W.Q0_DAY_LO, day_hi=W.Q0_DAY_HI):
    keep = ((c["day"] >= day_lo) & (c["day"] < day_hi) & (c["discount"] >= W.Q0_DISC_LO) & (c["discount"] <= W.Q0_DISC_HI)
            & (c["quantity"] < W.Q0_QTY))
    if mask is not None:
        keep &= mask
    return [[float((c["price"][keep] * c["discount"][keep]).sum()), int(keep.sum())]]


def _groupby_exact(c, mask, day_max=W.Q1_DAY):
    out = []
    dp = c["price"] * (1.0 - c["disc"])
    charge = dp * (1.0 + c["tax"])
    for a, b in W.GROUPS:
        keep = (c["flag_a"] == a) & (c["flag_b"] == b) & (c["day"] <= day_max)
        if mask is not None:
            keep &= mask
        n = int(keep.sum())
        s = [float(x[keep].sum()) for x in (c["qty"], c["price"], dp, charge, c["disc"])]
        avg = [x / n if n else math.nan for x in (s[0], s[1], s[4])]
        out.append(s[:4] + avg + [n])
    return out


def _join_exact(build, probe, day_lo=W.Q3_DAY_LO, day_hi=W.Q3_DAY_HI):
    keys, order = build["key"].sort()
    keep = (probe["day"] >= day_lo) & (probe["day"] < day_hi)
    fk, amount = probe["fk"][keep], probe["amount"][keep]
    at = torch.searchsorted(keys, fk).clamp_(max=len(keys) - 1)
    attr = torch.where(keys[at] == fk, build["attr"][order[at]], 99)
    return [[float(amount[attr == a].sum()), int((attr == a).sum())] for a in range(W.Q3_ATTR)]


def _as_answer(rows, case):
    """A Reduce's answer laid out as run() gives it."""
    if case["call"] == "launch":
        return {"fields": torch.tensor([r[:-1] for r in rows], dtype=torch.float64), "count": torch.tensor([r[-1] for r in rows])}
    return tuple(rows[0]) if case["kind"] == "filter_sum" else tuple(tuple(r) for r in rows)


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    n = case.get("rows", 0)
    if kind in ("filter_sum", "groupby"):
        cols = (_filter_sum_cols if kind == "filter_sum" else _groupby_cols)(g, n)
        mask = _mask(g, n, case["nulls"])
        return _as_answer((_filter_sum_exact if kind == "filter_sum" else _groupby_exact)(cols, mask), case)
    if kind == "join":
        return _as_answer(_join_exact(*_join_cols(g, case["build"], n)), case)
    if kind == "batch":
        tabs = []
        for shape, rows in _batch_shapes(case):
            if shape == "join":
                tabs.append(_join_cols(g, max(1000, rows // 20), rows))
            else:
                tabs.append(((_filter_sum_cols if shape == "filter_sum" else _groupby_cols)(g, rows), None))
        ask = {"filter_sum": _filter_sum_exact, "groupby": _groupby_exact, "join": _join_exact}
        fields, counts = [], []
        for k, shape, const in _batch_constants(case):
            for r in ask[shape](*tabs[k], **const):
                fields += r[:-1]
                counts.append(r[-1])
        return {"fields": np.array(fields, dtype=np.float64), "count": np.array(counts, dtype=np.int64)}
    if kind == "hashgroup":
        c, mult = _hash_cols(g, case)
        mask = _mask(g, n, case["nulls"])
        at = (c["key"] * pow(mult, -1, 1 << 40)) & ID_MASK
        ok = torch.ones(n, device="cuda", dtype=torch.bool) if mask is None else mask
        zero = lambda t: torch.zeros(case["keys"], device="cuda", dtype=t)  # noqa: E731
        return [zero(torch.int64).index_copy_(0, at, c["key"]),
                zero(torch.float64).index_add_(0, at, torch.where(ok, c["value"], 0.0)), zero(torch.int64).index_add_(0, at, ok.long())]
    if kind == "runs":
        keys, _, counts, vals = _run_cols(g, case)
        at = torch.repeat_interleave(torch.arange(len(keys), device="cuda"), counts)
        return [keys, torch.zeros(len(keys), device="cuda", dtype=torch.float64).index_add_(0, at, vals), counts]
    if kind == "select":
        c = _select_cols(g, n)
        keep = c["x"] < case["percent"]
        if case["vectorize"]:
            return [c["k"], c["x"] + 1, c["y"], None]
        return [c["k"][keep], c["x"][keep] + 1, c["y"][keep]]
    (ka, va), (kb, vb) = _merge_cols(g, case)
    # the j-th visit of a key pairs the j-th row of each side that holds it
    dup = 1 << 10
    code = [k * dup + torch.arange(len(k), device="cuda") - torch.searchsorted(k, k) for k in (ka, kb)]
    if case["mode"] == "inner":
        c = code[0][torch.isin(code[0], code[1])]
        c = c[c // dup <= min(int(ka[-1]), int(kb[-1]))]
        return [c // dup, va[torch.searchsorted(code[0], c)] + vb[torch.searchsorted(code[1], c)]]
    c = torch.unique(torch.cat(code))
    key, rank = c // dup, c % dup
    got = []
    for k, v in ((ka, va), (kb, vb)):
        lo = torch.searchsorted(k, key)
        row = lo + torch.minimum(rank, torch.searchsorted(k, key, right=True) - lo)
        got.append(torch.where(row < len(k), v[row.clamp(max=len(k) - 1)], torch.zeros((), dtype=v.dtype, device="cuda")))
    return [key, got[0] - got[1], got[0], got[1]]
