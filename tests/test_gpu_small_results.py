"""Small results at the edges of their paths: orders of up to 256 rows (by rank) and past it, gathers of up
to 1,024 rows in one launch and past it, strings that fill and overflow their 64 KB of room, batches read back
packed and column by column, NULLs around the 32- and 64-row words.  Row order and bytes are exact."""
import numpy as np
import pytest

from minilake_b200.abi import BOOL, COUNT, COUNT_STAR, DATE, FLOAT64, INT32, INT64, MAX, UTF8, AggSpec, Col, SortKey
from minilake_b200.columns import encode_strings, fixed, utf8_plain

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from minilake_b200.engine import GpuEngine
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield GpuEngine(ctx)
    ctx.close()


def _table(n, width=9):
    r = np.random.default_rng(n + width)
    text = [bytes(r.integers(97, 100, int(k), dtype=np.uint8)) for k in r.integers(0, width + 1, n)]
    ok = [r.random(n) > 0.2 for _ in range(6)]
    v = [r.integers(0, 5, n), np.round(r.normal(size=n), 1), r.integers(-9, 9, n), r.integers(0, 2, n), r.integers(0, 30, n)]
    cols = [fixed(INT64, v[0], ok[0]), fixed(FLOAT64, v[1]), fixed(INT32, v[2], ok[2]), fixed(BOOL, v[3], ok[3]),
            fixed(DATE, v[4]), utf8_plain(text, ok[5])]
    return cols, v, text, ok


def _same(got, cols, text, order):
    for g, w in zip(got, cols):
        m = w.valid_mask()[order]
        assert np.array_equal(g.valid_mask(), m)
        if w.dtype == UTF8:
            s = g.strings()
            assert all(s[i] == text[order[i]] for i in range(len(order)) if m[i])
        else:
            assert np.array_equal(g.values[m], w.values[order][m])


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("limit", [1, 7, None])
def test_orders_of_few_rows(engine, n, limit):
    cols, v, text, ok = _table(n)
    batch = engine.ctx.upload(cols)
    k = n if limit is None else min(limit, n)
    keys = [SortKey(Col(5), UTF8, asc=False, nulls_first=True), SortKey(Col(0), INT64)]
    rank = {t: i for i, t in enumerate(sorted(set(text)))}
    t = np.array([-rank[x] for x in text])
    order = np.lexsort([np.where(ok[0], v[0], 0), ~ok[0], np.where(ok[5], t, 0), ok[5]])[:k]
    for lim in (limit, n if limit is None else limit):  # the radix sort, and the top-N
        _same(engine.fetch(engine.topn(batch, batch.types, keys, lim)), cols, text, order)


@pytest.mark.parametrize("width", [63, 64, 65, 300])
def test_strings_around_their_room(engine, width):
    n = 1024  # of `width` bytes each: 64 KB at 64
    cols, v, text, ok = _table(n)
    text = [b"%04d" % i + b"x" * (width - 4) for i in range(n)]
    cols[5] = utf8_plain(text)
    batch = engine.ctx.upload(cols)
    order = np.lexsort([v[4]])
    _same(engine.fetch(engine.topn(batch, batch.types, [SortKey(Col(4), DATE)], n)), cols, text, order)


@pytest.mark.parametrize("groups", [0, 1, 6, 31, 33, 64, 65, 300, 5000])
def test_string_groups_and_values(engine, groups):
    """GROUP BY a dictionary string with a string MAX: ids become strings in one round trip."""
    r = np.random.default_rng(groups)
    n = groups * 9
    pool = [b"g%d" % i for i in range(groups)]
    idx = r.permutation(np.repeat(np.arange(groups), 9))
    w = [b"w%d" % i for i in range(50)]
    widx, ok = r.integers(0, 50, n), r.random(n) > 0.3
    batch = [encode_strings(pool, idx), utf8_plain([w[i] for i in widx], ok)]
    out = engine.fetch(engine.hashagg([batch], [UTF8, UTF8], [(Col(0), UTF8)],
                                      [AggSpec(COUNT_STAR), AggSpec(MAX, Col(1), UTF8), AggSpec(COUNT, Col(1), UTF8)]))
    got = dict(zip(out[0].strings(), zip(out[1].values.tolist(), [s if m else None for s, m in zip(out[2].strings(), out[2].valid_mask())],
                                         out[3].values.tolist())))
    want = {}
    for i in range(n):
        c, m, k = want.get(pool[idx[i]], (0, None, 0))
        x = w[widx[i]] if ok[i] else None
        want[pool[idx[i]]] = (c + 1, m if x is None else x if m is None else max(m, x), k + (x is not None))
    assert got == want
