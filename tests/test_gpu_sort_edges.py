"""ORDER BY at the edges of the device sort's units: tiles of 8,192 rows, keys of up to 32 varying bits
(sorted as they are), of more (sorted by the top 32, runs of equal keys put right) and keys whose top
32 bits tell few rows apart (every 32-bit piece sorted), over several words, types, orders and NULLs.
Row order is index work: the payload has to be numpy's stable order exactly."""
import numpy as np
import pytest

from minilake_b200.abi import DATE, FLOAT64, INT32, INT64, UTF8, Col, SortKey
from minilake_b200.columns import fixed, utf8_plain

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from minilake_b200.engine import GpuEngine
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield GpuEngine(ctx)
    ctx.close()


def _total(f):
    b = f.view(np.int64)
    return b ^ ((b >> 63).view(np.uint64) >> np.uint64(1)).view(np.int64)


def _case(kind, n):
    """Columns, sort keys, and numpy's keys, least significant first."""
    r = np.random.default_rng(n * 31 + len(kind))
    if kind == "few":  # 3 varying bits, most rows tied
        k = r.integers(0, 5, n)
        return [fixed(INT64, k)], [SortKey(Col(0), INT64, asc=False)], [-k]
    if kind == "same":
        return [fixed(INT64, np.full(n, 7))], [SortKey(Col(0), INT64)], [np.zeros(n)]
    if kind == "wide":  # 64 varying bits, told apart by the top 32 (and some that are not)
        k = r.integers(-(1 << 63), (1 << 63) - 1, n)
        k[r.random(n) < 0.05] = k[0]
        k = np.where(r.random(n) < 0.1, (k & ~np.int64(0xFF)) | r.integers(0, 4, n), k)
        return [fixed(INT64, k)], [SortKey(Col(0), INT64)], [k]
    if kind == "pieces":  # top 32 bits from four patterns: runs of a quarter of the rows
        k = (r.integers(-(1 << 31), 1 << 31, 4)[r.integers(0, 4, n)] << 32) | r.integers(0, 1 << 32, n)
        return [fixed(INT64, k)], [SortKey(Col(0), INT64, asc=False)], [-1 - k]
    if kind == "sparse":  # 30 varying bits spread over the word
        k = r.integers(0, 1 << 10, n) | (r.integers(0, 1 << 10, n) << 25) | (r.integers(0, 1 << 10, n) << 50)
        return [fixed(INT64, k)], [SortKey(Col(0), INT64)], [k]
    if kind == "two":  # a date, then an int32 descending with NULLs first
        d, v = r.integers(0, 40, n).astype(np.int32), r.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
        ok = r.random(n) > 0.2
        keys = [SortKey(Col(0), DATE), SortKey(Col(1), INT32, asc=False, nulls_first=True)]
        return [fixed(DATE, d), fixed(INT32, v, ok)], keys, [np.where(ok, -1 - v.astype(np.int64), 0), ok, d]
    if kind == "f64":
        f = np.round(r.normal(size=n) * 1e3, 1)
        f[r.random(n) < 0.05] = np.nan
        f[r.random(n) < 0.05] = -0.0
        f[r.random(n) < 0.05] = -np.inf
        ok = r.random(n) > 0.1
        return [fixed(FLOAT64, f, ok)], [SortKey(Col(0), FLOAT64)], [np.where(ok, _total(f), 0), ~ok]
    s = np.array([b"%016d" % x for x in r.integers(0, max(2, n // 3), n)])
    return [utf8_plain(list(s))], [SortKey(Col(0), UTF8)], [s]


@pytest.mark.parametrize("kind", ["few", "same", "wide", "pieces", "sparse", "two", "f64", "text"])
@pytest.mark.parametrize("n", [1, 2, 31, 8191, 8192, 8193, 24_581, 300_007])
def test_order_by_is_a_stable_sort(engine, kind, n):
    cols, keys, ref = _case(kind, n)
    batch = engine.ctx.upload(cols + [fixed(INT32, np.arange(n))])
    out = engine.fetch(engine.topn(batch, batch.types, keys, None))
    assert np.array_equal(out[-1].values, np.lexsort(ref))


def test_more_rows_than_the_prefix_sort_takes(engine):
    import torch
    from minilake_b200 import gpu
    n = (1 << 25) + 3
    k = np.random.default_rng(3).integers(-(1 << 63), (1 << 63) - 1, n)
    k[::7] &= ~np.int64(0xFFFFFFFF)
    batch = engine.ctx.upload([fixed(INT64, k), fixed(INT32, np.arange(n))])
    out = engine.topn(batch, batch.types, [SortKey(Col(0), INT64)], None)
    want = torch.sort(torch.from_numpy(k).cuda(), stable=True).indices
    assert torch.equal(gpu.column_tensor(out, 1).long(), want)
