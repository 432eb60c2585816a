"""The work a user has this framework do, as timed cases: queries over tables in HBM (as operator calls,
as a prepared query and through a serving loop's resident sinks), over host tables and over Parquet
files, and the operators a host engine calls one by one (filter, join probe, ORDER BY, top-N).

Shapes and distributions are those of the three benchmark queries (`minilake_b200/datagen.py`,
`workloads.py`, `serving.py`): filter + low-cardinality GROUP BY, join + high-cardinality GROUP BY +
top 10, star join with a string filter.  Tables reach from 100,000 rows to the 100M and 60M rows of
the benchmark's operators, with odd row counts and columns with NULLs among them.

`prepare` makes what a program holds before the call, on the GPU (host memory where the call takes
host tables or files); `run` is one call or query; `exact` gives the computed floating-point results
from plain torch or numpy.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from minilake_b200 import abi, datagen, gpu, parquet, workloads
from minilake_b200.abi import (AVG, BOOL, COUNT, COUNT_STAR, DATE, FLOAT64, INT32, INT64, MAX, MIN, SUM, UTF8, AggSpec,
                               Col, Lit, SortKey)
from minilake_b200.columns import HostColumn, fixed
from minilake_b200.engine import GpuEngine


def listed():
    return [
        # a serving slot's query: constants bound to a resident sink, graph replay, ORDER BY, result on the
        # host; the smallest table of the serving mix, where launches and host time count
        {"name": "serve_1m7", "kind": "serve", "rows": 1_700_017, "cutoff": 1200},
        # filter + GROUP BY two dictionary strings + four aggregates, the benchmark's 100M rows in HBM
        {"name": "filter_groupby_100m", "kind": "filter_groupby", "rows": 100_000_000, "morsels": 1, "cutoff": 2467,
         "nulls": False},
        # the headline query as a prepared plan: join 1.5M keys with 60M rows, GROUP BY the key, top 10
        {"name": "join_topn_60m", "kind": "join_topn", "rows": 60_000_000, "dim": 1_500_000, "cutoff": 1200},
        # the same query on host tables in pinned memory, 16 morsels pushed from 4 threads
        {"name": "join_host_4m", "kind": "join_host", "rows": 4_000_003, "dim": 1_500_000, "cutoff": 1200},
        # star join: LIKE on one dimension, three probes (Zipf keys), GROUP BY a build-side string; the
        # join tables are built in the query
        {"name": "star_join_60m", "kind": "star_join", "rows": 60_000_000, "prefix": "ab"},
        # GROUP BY a high-cardinality key through the hash table (no hint: it grows), every group out in
        # key order, one nullable argument
        {"name": "groupby_20m", "kind": "groupby", "rows": 20_000_003, "groups": 2_000_000, "wide": False, "nulls": True},
        # WHERE as an operator call: selection vector of 100M rows
        {"name": "filter_100m", "kind": "filter", "rows": 100_000_000, "cutoff": 2467, "nulls": False, "both": False},
        # join probe as an operator call: all (probe row, build row) pairs
        {"name": "probe_20m", "kind": "probe", "rows": 20_000_003, "build": 1_500_000, "sparse": False, "key": "i64"},
        # ORDER BY without a limit: a table of three columns by a DOUBLE, descending
        {"name": "order_by_10m", "kind": "order_by", "rows": 10_000_019, "keys": "f64"},
        # ORDER BY ... LIMIT 10 over the benchmark's 60M rows, and a result page of 100 rows
        {"name": "topn10_60m", "kind": "topn", "rows": 60_000_000, "limit": 10, "key": "f64", "nulls": False},
        {"name": "topn100_20m", "kind": "topn", "rows": 20_000_003, "limit": 100, "key": "f64", "nulls": False},
        # the filter + GROUP BY query from its Snappy Parquet file: 1M rows in 8 row groups, decoded on the GPU
        {"name": "parquet_1m", "kind": "parquet", "rows": 1_000_000, "row_groups": 8, "compression": "snappy"},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["serve", "filter_groupby", "join_topn", "join_host", "star_join", "groupby", "filter", "probe",
                       "order_by", "topn", "parquet"])
    cutoff = rng.randint(100, 2500)
    if kind == "serve":
        return {"kind": kind, "rows": log(100_000, 50_000_000), "cutoff": cutoff}
    if kind == "filter_groupby":
        return {"kind": kind, "rows": log(100_000, 100_000_000), "morsels": rng.choice([1, 1, 3, 8]), "cutoff": cutoff,
                "nulls": rng.random() < 0.4}
    if kind == "join_topn":
        return {"kind": kind, "rows": log(100_000, 60_000_000), "dim": log(10_000, 1_500_000), "cutoff": cutoff}
    if kind == "join_host":
        return {"kind": kind, "rows": log(100_000, 4_000_000), "dim": log(10_000, 1_500_000), "cutoff": cutoff}
    if kind == "star_join":
        return {"kind": kind, "rows": log(2_000_000, 60_000_000), "prefix": rng.choice(["ab", "q", "z", "th"])}
    if kind == "groupby":
        rows = log(100_000, 20_000_000)
        return {"kind": kind, "rows": rows, "groups": log(1_000, max(2_000, min(4_000_000, rows // 4))),
                "wide": rng.random() < 0.4, "nulls": rng.random() < 0.5}
    if kind == "filter":
        return {"kind": kind, "rows": log(100_000, 100_000_000), "cutoff": cutoff, "nulls": rng.random() < 0.4,
                "both": rng.random() < 0.4}
    if kind == "probe":
        return {"kind": kind, "rows": log(100_000, 20_000_000), "build": log(10_000, 1_500_000),
                "sparse": rng.random() < 0.5, "key": rng.choice(["i64", "i32"])}
    if kind == "order_by":
        return {"kind": kind, "rows": log(100_000, 10_000_000), "keys": rng.choice(["f64", "i64_nulls", "date_i32"])}
    if kind == "topn":
        return {"kind": kind, "rows": log(100_000, 60_000_000), "limit": log(1, 1_000),
                "key": rng.choice(["f64", "f64", "i64", "i32"]), "nulls": rng.random() < 0.3}
    return {"kind": kind, "rows": log(100_000, 1_500_000), "row_groups": rng.choice([1, 2, 4, 8]),
            "compression": rng.choice(["snappy", "snappy", "none"])}


def work(case):
    n, kind = case["rows"], case["kind"]
    if kind in ("serve", "filter_groupby"):  # d, two codes, three doubles; six groups come out
        b = 36 * n + (n // 8 if case.get("nulls") else 0)
    elif kind in ("join_topn", "join_host"):  # fk, d, v and the dimension's keys; ten rows come out
        b = 20 * n + 8 * case["dim"]
    elif kind == "star_join":  # k1 of every row, the rest of the rows that pass the first join, the dimensions
        b = 4 * n + 20 * n // 26 ** len(case["prefix"]) + 150_000 * 26 + 10_000 * 8 + 25 * 18
    elif kind == "groupby":
        b = (20 + (4 if case["wide"] else 0)) * n + (n // 8 if case["nulls"] else 0) + 48 * case["groups"]
    elif kind == "filter":
        keep = case["cutoff"] / 2557 * (0.5 if case["both"] else 1.0) * (0.9 if case["nulls"] else 1.0)
        b = (12 if case["both"] else 4) * n + (n // 8 if case["nulls"] else 0) + 4 * n * keep
    elif kind == "probe":  # the keys in, the pairs of the three in four rows that match out
        b = (8 if case["key"] == "i64" else 4) * (n + case["build"]) + 8 * n * 3 // 4
    elif kind == "order_by":
        b = 2 * {"f64": 20, "i64_nulls": 20, "date_i32": 20}[case["keys"]] * n
    elif kind == "topn":
        b = (4 if case["key"] == "i32" else 8) * n + (n // 8 if case["nulls"] else 0)
    else:  # the file's bytes (about 11 or 13 a row) in, the six columns out
        b = (36 + (11 if case["compression"] == "snappy" else 13)) * n
    return {"bytes": float(b), "flops": 0.0}


# ---- inputs --------------------------------------------------------------------------------------
_context = None


def _ctx():
    """The process's one context on the GPU, as a program that embeds the framework keeps it."""
    global _context
    if _context is None:
        _context = gpu.Context(0)
    return _context


def _random(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, n, lo, hi, dtype=torch.int32):
    return torch.randint(lo, hi, (n,), device="cuda", generator=g, dtype=dtype)


def _doubles(g, n, lo, hi):
    return torch.rand(n, device="cuda", generator=g, dtype=torch.float64) * (hi - lo) + lo


def _valid(g, n, share=0.9):
    return torch.rand(n, device="cuda", generator=g) < share


def _words(mask):
    """Validity words of a mask: bit i of the 64-bit words, lowest first."""
    n = mask.numel()
    m = torch.zeros((n + 63) // 64 * 64, dtype=torch.int64, device="cuda")
    m[:n] = mask
    return (m.view(-1, 64) << torch.arange(64, device="cuda")).sum(1)


class DeviceColumns:
    """Torch tensors as the columns of a device-resident batch: (type, tensor, validity mask or None,
    dictionary or None) each; `ml` is what the sinks and operators take."""

    def __init__(self, cols):
        n = cols[0][1].numel()
        arr = (abi.MlColumn * len(cols))()
        self.keep = []
        for i, (t, x, valid, dictionary) in enumerate(cols):
            arr[i].dtype, arr[i].location, arr[i].len, arr[i].data = t, abi.LOC_DEVICE, n, x.data_ptr()
            self.keep.append(x)
            if valid is not None:
                w = _words(valid)
                arr[i].validity = w.data_ptr()
                self.keep.append(w)
            if dictionary is not None:
                off = np.zeros(len(dictionary) + 1, dtype=np.uint32)
                np.cumsum([len(s) for s in dictionary], out=off[1:])
                data = np.frombuffer(b"".join(dictionary), dtype=np.uint8).copy()
                arr[i].encoding, arr[i].dict_len = abi.ENC_DICT, len(dictionary)
                arr[i].dict_offsets, arr[i].dict_data = off.ctypes.data, data.ctypes.data
                self.keep += [off, data]
        self.ml = (arr, len(cols), n)
        self.types = [c[0] for c in cols]


def _fg_columns(case, seed):
    """d, f1, f2, qty, price, disc and disc's validity mask, as datagen.filter_groupby distributes them."""
    n, g = case["rows"], _random(seed)
    d, f1, f2 = _ints(g, n, 0, 2557), _ints(g, n, 0, 3), _ints(g, n, 0, 2)
    qty = _ints(g, n, 1, 51, torch.int64).double()
    price = _ints(g, n, 90_000, 10_500_000, torch.int64).double() / 100.0
    disc = _ints(g, n, 0, 11, torch.int64).double() / 100.0
    return d, f1, f2, qty, price, disc, (_valid(g, n) if case.get("nulls") else None)


def _fg_batch(cols, part=slice(None)):
    d, f1, f2, qty, price, disc, valid = (None if c is None else c[part] for c in cols)
    return DeviceColumns([(INT32, d, None, None), (UTF8, f1, None, datagen.F1_VALUES), (UTF8, f2, None, datagen.F2_VALUES),
                          (FLOAT64, qty, None, None), (FLOAT64, price, None, None), (FLOAT64, disc, valid, None)])


def _join_columns(case, seed):
    """The dimension's keys (a permutation) and fk, d, v of the fact table, as datagen.join_groupby."""
    n, g = case["rows"], _random(seed)
    key = torch.randperm(case["dim"], device="cuda", generator=g) + 1
    return key, _ints(g, n, 1, case["dim"] + 1, torch.int64), _ints(g, n, 0, 2557), _doubles(g, n, 900.0, 105000.0)


A_ROWS, B_ROWS, C_ROWS = 150_000, 10_000, 25


def _strings(raw):
    """A plain string column of equally long strings (one row of bytes each)."""
    n, k = raw.shape
    return HostColumn(UTF8, np.ascontiguousarray(raw).reshape(-1), offsets=(np.arange(n + 1) * k).astype(np.uint32))


def _star_columns(case, seed):
    """Fact columns (k1 bounded Zipf(1.1) by inverse CDF, k2 uniform) and the three dimensions."""
    n, g = case["rows"], _random(seed)
    cdf = torch.cumsum(torch.arange(1, A_ROWS + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
    u = torch.rand(n, device="cuda", generator=g, dtype=torch.float64) * cdf[-1]
    k1 = (torch.searchsorted(cdf, u, right=True) + 1).clamp(1, A_ROWS).to(torch.int32)
    k2 = _ints(g, n, 1, B_ROWS + 1)
    v, w = _doubles(g, n, 0.0, 1e5), _doubles(g, n, 0.0, 0.1)
    r = np.random.default_rng(seed)
    a = (r.permutation(A_ROWS) + 1).astype(np.int32), r.integers(97, 123, (A_ROWS, 18), dtype=np.uint8)
    b = (r.permutation(B_ROWS) + 1).astype(np.int32), r.integers(0, C_ROWS, B_ROWS, dtype=np.int32)
    c = np.arange(C_ROWS, dtype=np.int32), r.integers(97, 123, (C_ROWS, 10), dtype=np.uint8)
    return (k1, k2, v, w), a, b, c


def _groupby_columns(case, seed):
    n, g = case["rows"], _random(seed)
    k = _ints(g, n, 0, case["groups"], torch.int64)
    k[torch.randperm(n, device="cuda", generator=g)[:case["groups"]]] = torch.arange(case["groups"], device="cuda")  # every group occurs
    k = k * 1_000_003 - (1 << 40)
    x, q = _doubles(g, n, -1000.0, 1000.0), _ints(g, n, 1, 51)
    day = (k % 7).to(torch.int32) + 10_000 if case["wide"] else None
    return k, day, x, q, (_valid(g, n) if case["nulls"] else None)


def _probe_columns(case, seed):
    """Distinct build keys (dense, or spread over 2^31) and probe keys of which three in four match."""
    g, t = _random(seed), (torch.int64 if case["key"] == "i64" else torch.int32)
    b = case["build"]
    build = torch.randperm(b, device="cuda", generator=g)
    row = _ints(g, case["rows"], 0, b + b // 3, torch.int64)
    step = max(1, (1 << 31) // (2 * b)) - 1 | 1 if case["sparse"] else 1
    return (build * step).to(t), (row * step).to(t)


def _order_columns(case, seed):
    n, g = case["rows"], _random(seed)
    payload = torch.arange(n, device="cuda", dtype=torch.int32)
    if case["keys"] == "f64":
        return [(FLOAT64, _doubles(g, n, 900.0, 105000.0), None, None), (INT64, _ints(g, n, 0, 1 << 40, torch.int64), None, None),
                (INT32, payload, None, None)]
    if case["keys"] == "i64_nulls":
        return [(INT64, _ints(g, n, -(1 << 20), 1 << 20, torch.int64), _valid(g, n), None), (FLOAT64, _doubles(g, n, 0.0, 1.0), None, None),
                (INT32, payload, None, None)]
    return [(DATE, _ints(g, n, 0, 2557), None, None), (INT32, _ints(g, n, 0, 1 << 30), None, None),
            (FLOAT64, _doubles(g, n, 0.0, 1.0), None, None), (INT32, payload, None, None)]


def _order_keys(case):
    if case["keys"] == "f64":
        return [SortKey(Col(0), FLOAT64, asc=False)]
    if case["keys"] == "i64_nulls":
        return [SortKey(Col(0), INT64)]
    return [SortKey(Col(0), DATE), SortKey(Col(1), INT32, asc=False)]


TOPN_TYPES = {"f64": FLOAT64, "i64": INT64, "i32": INT32}


def _topn_columns(case, seed):
    n, g = case["rows"], _random(seed)
    key = {"f64": lambda: _doubles(g, n, 900.0, 105000.0), "i64": lambda: _ints(g, n, -(1 << 62), 1 << 62, torch.int64),
           "i32": lambda: _ints(g, n, -(1 << 30), 1 << 30)}[case["key"]]()
    return key, (_valid(g, n) if case["nulls"] else None)


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = {"case": case, "ctx": ctx, "engine": GpuEngine(ctx)}
    if kind in ("serve", "filter_groupby"):
        cols = _fg_columns(case, seed)
        m, n = case.get("morsels", 1), case["rows"]
        step = (-(-n // m) + 63) // 64 * 64 if m > 1 else n  # row groups of whole validity words
        s["tables"] = [_fg_batch(cols, slice(a, min(a + step, n))) for a in range(0, n, step)]
        torch.cuda.synchronize()
        if kind == "serve":
            prologue, group, aggs = workloads.filter_groupby_plan(case["cutoff"])
            s["sink"] = gpu.HashAggregateSink(ctx, s["tables"][0].types, group, aggs, prologue)
    elif kind == "join_topn":
        key, fk, d, v = _join_columns(case, seed)
        s["dim"] = DeviceColumns([(INT64, key, None, None)])
        s["fact"] = DeviceColumns([(INT64, fk, None, None), (INT32, d, None, None), (FLOAT64, v, None, None)])
        torch.cuda.synchronize()
        q = gpu.Query(ctx)
        table = q.add_build(gpu.JoinBuildSink(ctx, [INT64], [(Col(0), INT64)]), s["dim"].ml)
        prologue, group, aggs = workloads.join_groupby_plan(table, case["cutoff"])
        q.set_aggregate(gpu.HashAggregateSink(ctx, s["fact"].types, group, aggs, prologue), s["fact"].ml)
        q.set_topn(workloads.join_groupby_topn_keys(), 10)
        q.run_host()  # the planning run
        s["query"] = q
    elif kind == "join_host":
        cols = [c.cpu().pin_memory() for c in _join_columns(case, seed)]
        s["pinned"] = cols
        key, fk, d, v = (c.numpy() for c in cols)
        at = np.linspace(0, case["rows"], 17).astype(np.int64)
        s["dim"] = [fixed(INT64, key)]
        s["fact"] = [[fixed(INT64, fk[a:b]), fixed(INT32, d[a:b]), fixed(FLOAT64, v[a:b])] for a, b in zip(at, at[1:])]
        s["engine"] = GpuEngine(ctx, threads=4)
    elif kind == "star_join":
        (k1, k2, v, w), a, b, c = _star_columns(case, seed)
        s["fact"] = DeviceColumns([(INT32, k1, None, None), (INT32, k2, None, None), (FLOAT64, v, None, None),
                                   (FLOAT64, w, None, None)])
        s["A"] = ctx.upload([fixed(INT32, a[0]), _strings(a[1])])
        s["B"] = ctx.upload([fixed(INT32, b[0]), fixed(INT32, b[1])])
        s["C"] = ctx.upload([fixed(INT32, c[0]), _strings(c[1])])
    elif kind == "groupby":
        k, day, x, q, valid = _groupby_columns(case, seed)
        s["table"] = DeviceColumns([(INT64, k, None, None), (FLOAT64, x, valid, None), (INT32, q, None, None)] +
                                   ([(DATE, day, None, None)] if case["wide"] else []))
    elif kind == "filter":
        d, _, _, _, price, _, valid = _fg_columns(case, seed)
        s["table"] = DeviceColumns([(INT32, d, valid, None), (FLOAT64, price, None, None)])
        s["sel"] = torch.zeros(case["rows"], dtype=torch.int32, device="cuda")
    elif kind == "probe":
        build, row = _probe_columns(case, seed)
        t = INT64 if case["key"] == "i64" else INT32
        s["dim"], s["table"] = DeviceColumns([(t, build, None, None)]), DeviceColumns([(t, row, None, None)])
        torch.cuda.synchronize()
        s["join"] = s["engine"].join_build([s["dim"].ml], [t], [(Col(0), t)])
        s["pairs"] = [torch.zeros(case["rows"], dtype=torch.int32, device="cuda") for _ in range(2)]
    elif kind == "order_by":
        s["table"] = DeviceColumns(_order_columns(case, seed))
    elif kind == "topn":
        key, valid = _topn_columns(case, seed)
        s["table"] = DeviceColumns([(TOPN_TYPES[case["key"]], key, valid, None)])
    else:
        s["dir"] = tempfile.TemporaryDirectory()
        s["path"] = os.path.join(s["dir"].name, "t.parquet")
        datagen.filter_groupby_parquet(s["path"], rows=case["rows"], row_groups=case["row_groups"], seed=seed,
                                       compression=case["compression"])
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------------------------
def _host(cols):
    """Fetched result columns as arrays, by column number."""
    out = {}
    for i, c in enumerate(cols):
        out["c%d" % i] = c.values
        if c.offsets is not None:
            out["c%d_offsets" % i] = c.offsets
        if c.validity is not None:
            out["c%d_valid" % i] = c.validity
    return out


class _Words:
    """A device batch's validity words, for torch."""

    def __init__(self, ptr, words, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (words,), "typestr": "<i8", "data": (ptr, False), "version": 3}


def _device(batch):
    """A device batch's columns as tensors (views; the batch lives as long as they do)."""
    out, (arr, n), rows = {}, batch.ml_columns(), batch.num_rows
    for i in range(n):
        out["c%d" % i] = gpu.column_tensor(batch, i)
        if arr[i].validity and rows:
            out["c%d_valid" % i] = torch.as_tensor(_Words(arr[i].validity, (rows + 63) // 64, batch), device="cuda")
    return out


def _sort(ctx, types, keys, limit, batch):
    sink = gpu.SortSink(ctx, types, keys, limit)
    local = sink.create_local()
    local.sink(batch)
    local.combine()
    out = sink.finalize()
    sink.close()
    return out


def run(s):
    case, ctx, engine = s["case"], s["ctx"], s["engine"]
    kind = case["kind"]
    if kind == "serve":
        s["sink"].rebind(*workloads.filter_groupby_plan(case["cutoff"]))
        s["sink"].run_resident(s["tables"][0].ml, reset=True)
        agg = s["sink"].finalize()
        keys = [SortKey(Col(0), UTF8), SortKey(Col(1), UTF8)]
        return _host(_sort(ctx, workloads.FG_OUT_TYPES, keys, max(agg.num_rows, 1), agg).fetch())
    if kind == "filter_groupby":
        return _host(workloads.run_filter_groupby(engine, [t.ml for t in s["tables"]], case["cutoff"]))
    if kind == "join_topn":
        return _host(s["query"].run_host())
    if kind == "join_host":
        return _host(workloads.run_join_groupby(engine, [s["dim"]], s["fact"], case["cutoff"]))
    if kind == "star_join":
        builds = workloads.star_join_builds(engine, s["A"], s["B"], s["C"], case["prefix"] + "%")
        return _host(workloads.run_star_join(engine, [s["fact"].ml], s["A"], s["B"], s["C"], builds=builds))
    if kind == "groupby":
        wide = case["wide"]
        group = [(Col(0), INT64)] + ([(Col(3), DATE)] if wide else [])
        aggs = [AggSpec(SUM, Col(1), FLOAT64), AggSpec(AVG, Col(1), FLOAT64), AggSpec(COUNT, Col(1), FLOAT64),
                AggSpec(SUM, Col(2), INT64), AggSpec(MIN, Col(1), FLOAT64), AggSpec(MAX, Col(2), INT32), AggSpec(COUNT_STAR)]
        agg = engine.hashagg([s["table"].ml], s["table"].types, group, aggs)
        types = agg.types
        keys = [SortKey(Col(0), INT64)] + ([SortKey(Col(1), DATE)] if wide else [])
        return _device(engine.topn(agg, types, keys, None))
    if kind == "filter":
        pred = Col(0) <= Lit(case["cutoff"])
        if case["both"]:
            pred = pred & (Col(1) < Lit(52_950.0))
        keep = abi.Keep()
        e = abi.encode_expr(pred, BOOL, keep)
        (arr, nc, n), k = s["table"].ml, ctypes.c_int64()
        gpu._check(gpu.LIB.ml_gpu_filter(ctx.h, ctypes.byref(e), arr, nc, n, None, 0, abi.LOC_DEVICE, s["sel"].data_ptr(),
                                         ctypes.byref(k)))
        return [s["sel"], k.value]  # the caller's buffer, and how many entries of it count
    if kind == "probe":
        keep = abi.Keep()
        t = INT64 if case["key"] == "i64" else INT32
        e, ne = abi.encode_exprs([(Col(0), t)], keep)
        (arr, nc, n), k = s["table"].ml, ctypes.c_int64()
        gpu._check(gpu.LIB.ml_gpu_join_probe(ctx.h, s["join"].handle, e, ne, arr, nc, n, None, 0, abi.LOC_DEVICE,
                                             s["pairs"][0].data_ptr(), s["pairs"][1].data_ptr(), case["rows"], ctypes.byref(k)))
        return s["pairs"] + [k.value]  # the caller's buffers, and how many entries of them count
    if kind == "order_by":
        return _device(engine.topn([s["table"].ml], s["table"].types, _order_keys(case), None))
    if kind == "topn":
        t = s["table"].types
        return _host(engine.topn([s["table"].ml], t, [SortKey(Col(0), t[0], asc=False)], case["limit"]).fetch())
    morsels = parquet.read_table(ctx, s["path"], workloads.FG_SCAN)
    out = _host(workloads.run_filter_groupby(engine, [m.ml for m in morsels]))
    for name, i in (("d", 0), ("qty", 3), ("price", 4), ("disc", 5)):
        out[name] = [gpu.column_tensor(m.batches[i], 0) for m in morsels]
    return out


# ---- what the floating-point results are, in 64 bits -----------------------------------------------
def _fg_exact(d, f1, f2, qty, price, disc, ok, cutoff):
    """SUM(qty), SUM(price * (1 - disc)), AVG(disc) per (f1, f2) in key order; ok: where disc is not NULL."""
    sums = [[], [], []]
    for a in range(3):
        for b in range(2):
            m = (d <= cutoff) & (f1 == a) & (f2 == b)
            if not bool(m.any()):
                continue
            v = m & ok
            sums[0].append(float(qty[m].sum()))
            sums[1].append(float((price[v] * (1 - disc[v])).sum()))
            sums[2].append(float(disc[v].sum()) / max(int(v.sum()), 1))
    return {"c%d" % (2 + i): np.array(x) for i, x in enumerate(sums)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("serve", "filter_groupby"):
        *cols, valid = _fg_columns(case, seed)
        return _fg_exact(*cols, torch.ones_like(cols[0], dtype=torch.bool) if valid is None else valid, case["cutoff"])
    if kind in ("join_topn", "join_host"):
        _, fk, d, v = _join_columns(case, seed)
        keep = d > case["cutoff"]
        s = torch.zeros(case["dim"] + 1, dtype=torch.float64, device="cuda").index_add_(0, fk[keep], v[keep])
        return {"c1": torch.topk(s, 10).values}
    if kind == "star_join":
        (k1, k2, v, w), a, b, _ = _star_columns(case, seed)
        p = np.frombuffer(case["prefix"].encode(), dtype=np.uint8)
        match = torch.zeros(A_ROWS + 1, dtype=torch.bool, device="cuda")
        match[torch.from_numpy(a[0][(a[1][:, :len(p)] == p).all(1)].astype(np.int64)).cuda()] = True
        region = torch.zeros(B_ROWS + 1, dtype=torch.int64, device="cuda")
        region[torch.from_numpy(b[0].astype(np.int64)).cuda()] = torch.from_numpy(b[1].astype(np.int64)).cuda()
        m = match[k1.long()]
        s = torch.zeros(C_ROWS, dtype=torch.float64, device="cuda")
        s.index_add_(0, region[k2[m].long()], v[m] * (1 - w[m]))
        return {"c1": torch.sort(s[s > 0], descending=True).values}
    if kind == "groupby":
        k, _, x, _, valid = _groupby_columns(case, seed)
        u, inv = torch.unique(k, return_inverse=True)
        ok = valid if valid is not None else torch.ones_like(k, dtype=torch.bool)
        s = torch.zeros(u.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv[ok], x[ok])
        c = torch.bincount(inv[ok], minlength=u.numel())
        lo = torch.zeros_like(s).scatter_reduce_(0, inv[ok], x[ok], "amin", include_self=False)
        at = 2 if case["wide"] else 1
        return {"c%d" % at: s, "c%d" % (at + 1): torch.where(c > 0, s / c.clamp(min=1), 0.0), "c%d" % (at + 4): lo}
    if kind == "topn" and case["key"] == "f64":
        key, valid = _topn_columns(case, seed)
        return {"c0": torch.topk(key if valid is None else key[valid], case["limit"]).values}
    if kind == "parquet":  # the values datagen.filter_groupby_parquet writes
        n, r = case["rows"], np.random.Generator(np.random.PCG64(seed))
        d, f1, f2 = r.integers(0, 2557, n, dtype=np.int32), r.integers(0, 3, n), r.integers(0, 2, n)
        qty = r.integers(1, 51, n).astype(np.float64)
        price, disc = r.integers(90_000, 10_500_000, n) / 100.0, r.integers(0, 11, n) / 100.0
        return _fg_exact(d, f1, f2, qty, price, disc, np.ones(n, dtype=bool), 2467)
    return None  # selections, join pairs and reordered rows compute no numbers
