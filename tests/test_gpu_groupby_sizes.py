"""GROUP BY without a size hint over batches large enough to be taken in ranges (65,536 rows, then the
rest, or ranges of growing size), at the edges of the table's and the kernel's cases: few groups, around
the 1,024 the table starts with, groups that keep coming at the end of the batch, nearly one per row,
skewed; one- and two-word keys with NULLs; every accumulator, with and without NULL arguments, through
the warp-cooperative updates.  Counts, integer sums, minima and maxima have to be numpy's exactly; f64 sums are
compared with exactly rounded ones, within n * 2^-53 of the sum of magnitudes (n additions in any order)."""
import numpy as np
import pytest

from minilake_b200.abi import (AVG, COUNT, COUNT_STAR, FLOAT64, INT32, INT64, MAX, MIN, SUM, AggSpec, Col)
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from minilake_b200.engine import GpuEngine
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield GpuEngine(ctx)
    ctx.close()


def _keys(kind, n, r):
    if kind == "few":
        return r.integers(0, 7, n)
    if kind == "quarter":  # just above a quarter of the first table
        return r.integers(0, 257, n)
    if kind == "table":
        return r.integers(0, 1025, n)
    if kind == "late":  # 40 groups, then a new one per row
        return np.where(np.arange(n) < n - 90_000, r.integers(0, 40, n), np.arange(n))
    if kind == "clustered":
        return np.arange(n) // 3
    if kind == "distinct":
        return r.permutation(n)
    return np.minimum((1 / np.maximum(r.random(n), 1e-12)).astype(np.int64), 1 << 40)  # skewed


AGGS = [AggSpec(COUNT_STAR), AggSpec(SUM, Col(1), FLOAT64), AggSpec(AVG, Col(1), FLOAT64), AggSpec(COUNT, Col(1), FLOAT64),
        AggSpec(SUM, Col(2), INT64), AggSpec(MIN, Col(1), FLOAT64), AggSpec(MAX, Col(2), INT64), AggSpec(MIN, Col(2), INT64)]


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("kind", ["few", "quarter", "table", "late", "clustered", "distinct", "skewed"])
@pytest.mark.parametrize("n", [262_143, 262_144, 700_001])
def test_groups_of_every_number(engine, kind, n, nulls, wide):
    r = np.random.default_rng(n + len(kind))
    k = _keys(kind, n, r)
    k2 = (k % 5).astype(np.int32)
    kv = r.random(n) > 0.01 if nulls else np.ones(n, dtype=bool)
    x, q = np.round(r.normal(size=n) * 1e3, 2), r.integers(-(1 << 40), 1 << 40, n)
    xv = r.random(n) > 0.2 if nulls else np.ones(n, dtype=bool)
    mask = lambda m: m if nulls else None  # noqa: E731
    cols = [fixed(INT64, k * 977 - (1 << 33), mask(kv)), fixed(FLOAT64, x, mask(xv)), fixed(INT64, q)]
    group = [(Col(0), INT64)]
    if wide:
        cols.append(fixed(INT32, k2))
        group.append((Col(3), INT32))
    batch = engine.ctx.upload(cols)
    out = engine.hashagg([batch], batch.types, group, AGGS)
    got = engine.fetch(out)
    nk = len(group)
    # the groups as one code each: the key, or a code of its own for NULL (with k2 beside it)
    code = np.where(kv, k, np.int64(1) << 62)
    if wide:
        code = code + (np.where(kv, np.int64(0), k2.astype(np.int64)))
    u, inv = np.unique(code, return_inverse=True)
    gk = np.where(got[0].valid_mask(), (got[0].values + (1 << 33)) // 977, np.int64(1) << 62)
    if wide:
        gk = gk + np.where(got[0].valid_mask(), 0, got[1].values.astype(np.int64))
    order = np.argsort(gk)
    assert np.array_equal(gk[order], u)
    a = [c for c in got[nk:]]
    m = len(u)
    cnt, cx = np.bincount(inv, minlength=m), np.bincount(inv[xv], minlength=m)
    has = cx > 0
    assert np.array_equal(a[0].values[order], cnt) and np.array_equal(a[3].values[order], cx)
    # exactly rounded sums: the values are whole cents, their sums exact in integers
    cents = np.zeros(m, dtype=np.int64)
    np.add.at(cents, inv[xv], np.rint(x[xv] * 100).astype(np.int64))
    mag = np.bincount(inv[xv], weights=np.abs(x[xv]), minlength=m)
    # each x is cents / 100 rounded once, the sum adds at most cnt roundings
    tol = (cnt + 2) * 2.0 ** -53 * mag * 1.0001
    assert np.array_equal(a[1].valid_mask()[order], has)
    assert np.all(np.abs(a[1].values[order] - cents / 100)[has] <= tol[has])
    assert np.all(np.abs(a[2].values[order] - cents / 100 / np.maximum(cx, 1))[has] <= 2 * tol[has] / cx[has])
    qs = np.zeros(m, dtype=np.int64)
    np.add.at(qs, inv, q)
    assert np.array_equal(a[4].values[order], qs)
    lo = np.full(m, np.inf)
    np.minimum.at(lo, inv[xv], x[xv])
    assert np.array_equal(a[5].valid_mask()[order], has) and np.array_equal(a[5].values[order][has], lo[has])
    hi, low = np.full(m, -(1 << 62)), np.full(m, 1 << 62)
    np.maximum.at(hi, inv, q)
    np.minimum.at(low, inv, q)
    assert np.array_equal(a[6].values[order], hi) and np.array_equal(a[7].values[order], low)


@pytest.mark.parametrize("build", [40, 70_000])
def test_join_groups_share_a_sector(engine, build):
    """GROUP BY the join key: the count and the sum of a group are updated by a pair of lanes (through
    global memory for 70,000 build rows; the first 256 of 40 in shared memory)."""
    from minilake_b200 import workloads
    from minilake_b200.columns import Table
    from oracle import orc
    r = np.random.default_rng(build)
    n = 400_003
    dim = [fixed(INT64, r.permutation(build).astype(np.int64))]
    fact = [fixed(INT64, r.integers(0, build + 9, n)), fixed(INT32, r.integers(0, 2557, n).astype(np.int32)),
            fixed(FLOAT64, np.round(r.random(n) * 1e5, 2))]
    got = workloads.run_join_groupby(engine, Table("dim", ["key"], [dim]), Table("fact", ["fk", "d", "v"], [fact]), limit=30)
    want = workloads.run_join_groupby(orc.OracleEngine(threads=2), Table("dim", ["key"], [dim]),
                                      Table("fact", ["fk", "d", "v"], [fact]), limit=30)
    assert np.array_equal(got[0].values, want[0].values) and np.array_equal(got[2].values, want[2].values)
    assert np.abs(got[1].values - want[1].values).max() <= 1e-12 * np.abs(want[1].values).max()
