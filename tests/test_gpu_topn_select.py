"""ORDER BY ... LIMIT by selection (a sampled bound, a pass that lists the rows at or below it, the exact
k-th) at its edges: the row counts where it starts, the smallest and largest limits, every fixed-width
type, both orders, NULLs first and last and NULL only, ties at the limit within and past what the final
sort holds, a column whose sample misleads (sorted, periodic).  Row order is index work: the rows kept
have to be the first of numpy's stable sort exactly."""
import numpy as np
import pytest

from minilake_b200.abi import BOOL, DATE, FLOAT64, INT32, INT64, Col, SortKey
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield ctx
    ctx.close()


def _check(ctx, dtype, v, valid, limit, asc, nulls_first):
    from minilake_b200.engine import GpuEngine
    n = len(v)
    batch = ctx.upload([fixed(dtype, v, valid), fixed(INT32, np.arange(n))])
    eng = GpuEngine(ctx)
    out = eng.fetch(eng.topn(batch, batch.types, [SortKey(Col(0), dtype, asc=asc, nulls_first=nulls_first)], limit))
    key = v.astype(np.float64 if dtype == FLOAT64 else np.int64)
    if dtype == FLOAT64:
        b = key.view(np.int64)
        key = b ^ ((b >> 63).view(np.uint64) >> np.uint64(1)).view(np.int64)
    key = key if asc else -1 - key
    ok = np.ones(n, dtype=bool) if valid is None else valid
    order = np.lexsort([np.where(ok, key, 0), ok if nulls_first else ~ok])
    assert np.array_equal(out[1].values, order[:limit])


@pytest.mark.parametrize("limit", [33, 100, 2048])
@pytest.mark.parametrize("n", [2048, 65_535, 65_536, 65_537, 300_001])
@pytest.mark.parametrize("dtype", [FLOAT64, INT64, INT32, DATE])
def test_limits_by_selection(ctx, dtype, n, limit):
    r = np.random.default_rng(n + limit)
    v = np.round(r.normal(size=n) * 1e6) / 7 if dtype == FLOAT64 else r.integers(-(1 << 30), 1 << 30, n)
    if dtype == FLOAT64:
        v[r.random(n) < 0.001] = np.nan
        v[r.random(n) < 0.001] = -np.inf
        v[r.random(n) < 0.001] = -0.0
    valid = r.random(n) > 0.1 if limit == 100 else None
    _check(ctx, dtype, v, valid, limit, bool(n & 1), dtype == INT32)


@pytest.mark.parametrize("limit", [1, 10, 32])
@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21, 2_500_003])
def test_small_limits_over_many_rows(ctx, n, limit):
    r = np.random.default_rng(n + limit)
    _check(ctx, FLOAT64, r.random(n), None, limit, False, False)
    _check(ctx, INT32, r.integers(0, 1 << 30, n), r.random(n) > 0.5, limit, True, True)


@pytest.mark.parametrize("kind", ["sorted", "reversed", "periodic", "ties", "more_ties", "null_only", "bool"])
@pytest.mark.parametrize("limit", [40, 2048])
def test_columns_that_mislead(ctx, kind, limit):
    n = 400_000
    r = np.random.default_rng(5)
    v, valid, dtype = np.arange(n), None, INT64
    if kind == "reversed":
        v = v[::-1].copy()
    if kind == "periodic":  # small values only at every 24th row
        v = np.where(v % 24 == 3, v, v + (1 << 40))
    if kind == "ties":  # about 3,000 rows at the limit
        v = r.integers(0, n // 3000, n)
    if kind == "more_ties":  # 100,000
        v = r.integers(0, 4, n)
    if kind == "null_only":
        valid = np.zeros(n, dtype=bool)
    if kind == "bool":
        v, dtype = r.integers(0, 2, n), BOOL
    _check(ctx, dtype, v, valid, limit, True, False)
