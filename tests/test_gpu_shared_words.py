"""Aggregates over one argument share accumulator words (AVG's sum and count serve SUM and COUNT, a count
tells SUM, MIN and MAX whether they saw a value): every combination and order has to give what each
aggregate gives alone, with and without NULLs, over casts, with NULLs that appear only in a later batch,
grouped (few groups, many groups) and not, specialized and interpreted.  Inputs are whole numbers
below 2^20 and there are fewer than 2^20 rows, so f64 sums are exact and everything is compared exactly."""
import itertools

import numpy as np
import pytest

from minilake_b200.abi import (AVG, COUNT, COUNT_STAR, FLOAT64, INT32, INT64, MAX, MIN, SUM, AggSpec, Col, Lit)
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu

X = (Col(1), FLOAT64)
I = (Col(2), INT32)
L = (Col(1) * Lit(2.0), FLOAT64)  # a literal: never shared, same results
SETS = [list(c) for c in itertools.permutations([(SUM, X), (AVG, X), (COUNT, X), (MIN, X)])] + [
    [(SUM, X), (MIN, X), (MAX, X), (SUM, X), (MIN, X)],
    [(MIN, X), (MIN, X), (SUM, X)],
    [(COUNT, X), (COUNT, X), (MAX, X), (COUNT_STAR, None)],
    [(AVG, X), (AVG, X), (COUNT, X), (SUM, X)],
    [(AVG, I), (COUNT, I), (SUM, I), (MIN, I), (MAX, I), (AVG, X), (MAX, X)],
    [(SUM, I), (MIN, I), (SUM, I)],
    [(SUM, L), (AVG, L), (COUNT, L), (AVG, X)],
]


def _want(func, arg, sel, x, xv, i, iv):
    if func == COUNT_STAR:
        return int(sel.sum())
    v, ok = (i, iv) if arg is I else (x * 2 if arg is L else x, xv)
    v = v[sel & ok]
    if func == COUNT:
        return len(v)
    if not len(v):
        return None
    if func == SUM:
        return v.sum()
    if func == AVG:
        return float(v.sum()) / len(v)
    return v.min() if func == MIN else v.max()


@pytest.mark.parametrize("flags", [0, 4], ids=["specialized", "interpreted"])
@pytest.mark.parametrize("groups", [0, 5, 3000])
@pytest.mark.parametrize("nulls", ["none", "late", "all"])
def test_aggregates_of_one_argument(flags, groups, nulls):
    from minilake_b200 import gpu
    from minilake_b200.engine import GpuEngine
    ctx = gpu.Context(0, flags=flags)
    engine = GpuEngine(ctx)
    r = np.random.default_rng(groups + len(nulls))
    n = 40_000
    k = r.integers(0, max(groups, 1), n)
    x, i = r.integers(-(1 << 20), 1 << 20, n).astype(np.float64), r.integers(-(1 << 20), 1 << 20, n, dtype=np.int32)
    xv, iv = np.ones(n, dtype=bool), np.ones(n, dtype=bool)
    half = n // 2
    if nulls != "none":
        s = slice(half, n) if nulls == "late" else slice(0, n)
        xv[s], iv[s] = r.random(s.stop - s.start) > 0.3, r.random(s.stop - s.start) > 0.3
        if groups:  # groups without a single value
            xv[k % 5 == 3] = False
            if nulls == "late":
                xv[:half] = True
    batches = []
    for s in (slice(0, half), slice(half, n)):
        m = lambda v: None if v[s].all() else v[s]  # noqa: E731
        batches.append(ctx.upload([fixed(INT64, k[s]), fixed(FLOAT64, x[s], m(xv)), fixed(INT32, i[s], m(iv))]))
    check = np.unique(k)[:: max(1, groups // 40)] if groups else [0]
    for aggs in SETS:
        specs = [AggSpec(f) if a is None else AggSpec(f, *a) for f, a in aggs]
        out = engine.fetch(engine.hashagg(batches, batches[0].types, [(Col(0), INT64)] if groups else [], specs))
        cols = out[1:] if groups else out
        where = {int(v): j for j, v in enumerate(out[0].values)} if groups else {0: 0}
        assert len(where) == (len(np.unique(k)) if groups else 1)
        for g in check:
            sel = k == g if groups else np.ones(n, dtype=bool)
            for (f, a), c in zip(aggs, cols):
                want, j = _want(f, a, sel, x, xv, i, iv), where[int(g)]
                valid = c.validity is None or c.valid_mask()[j]
                assert valid == (want is not None), (aggs, f, g)
                if valid:
                    assert c.values[j] == want, (aggs, f, g, c.values[j], want)
    ctx.close()
