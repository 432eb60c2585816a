"""Filters and aggregates over pageable host columns from many threads of one context, as MiniLake's workers
call them: the columns' widths grow (INT32, a dictionary string, DOUBLE with NULLs), so every thread's
pinned staging block is replaced while copies are in flight.  Each result has to equal the same call made
alone (row ids, counts and sums of whole numbers: identical)."""
import threading

import numpy as np
import pytest

from minilake_b200.abi import COUNT, COUNT_STAR, FLOAT64, INT32, INT64, MIN, SUM, UTF8, AggSpec, Col, Lit
from minilake_b200.columns import encode_strings, fixed

pytestmark = pytest.mark.gpu

POOL = [b"a", b"bb", b"ccc", b"dddd", b"eeeee"]


def _batch(t):
    r = np.random.default_rng(100 + t)
    n = 40_000 + 7_001 * t
    return [fixed(INT32, r.integers(0, 1000, n)), encode_strings(POOL[: 3 + t % 3], r.integers(0, 3 + t % 3, n)),
            fixed(FLOAT64, r.integers(0, 1 << 20, n).astype(np.float64), r.random(n) > 0.2),
            fixed(INT64, r.integers(0, 1 << 40, n), r.random(n) > 0.1)]


def test_eight_threads_with_growing_pageable_columns():
    from minilake_b200.gpu import Context, FilterOperator, HashAggregateSink
    batches = [_batch(t) for t in range(8)]

    def work(ctx, cols):
        sel = FilterOperator(ctx, (Col(2) > Lit(1000.0)) & (Col(0) < Lit(900))).execute(cols)
        sink = HashAggregateSink(ctx, [INT32, UTF8, FLOAT64, INT64], [(Col(1), UTF8)],
                                 [AggSpec(COUNT_STAR), AggSpec(COUNT, Col(2), FLOAT64), AggSpec(SUM, Col(2), FLOAT64),
                                  AggSpec(MIN, Col(3), INT64), AggSpec(SUM, Col(0), INT32)])
        loc = sink.create_local()
        for _ in range(2):
            loc.sink(cols)
            loc.sink(cols, sel)
        loc.combine()
        b = sink.finalize()
        out = b.fetch()
        b.close()
        sink.close()
        keys = out[0].strings()
        order = np.argsort(keys)
        return sel, [keys[i] for i in order], [c.values[order] for c in out[1:]]

    with_one = Context(0)
    alone = [work(with_one, b) for b in batches]
    with_one.close()
    ctx = Context(0)  # fresh: its pool of pinned blocks is empty
    wrong, errors = [], []

    def run(i):
        try:
            for _ in range(10):
                sel, keys, vals = work(ctx, batches[i])
                a = alone[i]
                if not (np.array_equal(sel, a[0]) and keys == a[1] and all(np.array_equal(x, y) for x, y in zip(vals, a[2]))):
                    wrong.append(i)
        except BaseException as e:  # reported below
            errors.append(e)

    ts = [threading.Thread(target=run, args=(i,)) for i in range(len(batches))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    ctx.close()
    assert not errors, errors
    assert not wrong, wrong
