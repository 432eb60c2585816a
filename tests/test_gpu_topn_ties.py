"""ORDER BY ... LIMIT where many rows share the first key at the limit (few distinct values, NULLs in front,
the type's lowest value beside them) and the NULL flags, the other keys or the row order decide: the rows kept
are a stable sort's, and the selection finds them (no other route is timed after it).  Row counts on both sides
of the selection's direct form and of its two sample sizes."""
import numpy as np
import pytest

from minilake_b200.abi import BOOL, FLOAT64, INT32, INT64, UTF8, Col, SortKey
from minilake_b200.columns import fixed, utf8_plain

pytestmark = pytest.mark.gpu

POOL = sorted([b"", b"\0", b"a", b"a\0", b"a\0\0\0\0\0\0\0\0b", b"common prefix of", b"common prefix of\0", b"common prefix of the", b"common prefix of thf",
               b"common prefix og", b"common prefix of all the longer strings 0", b"common prefix of all the longer strings 1"])
SIZES = [(60_001, 40), (60_001, 2048), (65_537, 33), (400_003, 100), (400_003, 2048), ((1 << 21) + 1, 1), ((1 << 21) + 1, 32), (4_200_005, 10),
         (4_200_005, 1500)]


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200.gpu import PROFILE, Context
    ctx = Context(0, flags=PROFILE)
    yield ctx
    ctx.close()


def _columns(n, seed):
    """name -> (column, dtype, value order, valid)"""
    r = np.random.default_rng(seed)
    four = r.integers(0, 4, n)
    days = np.sort(r.integers(0, 50, n))
    half = r.random(n) < 0.5
    low = np.where(r.random(n) < 0.3, np.iinfo(np.int64).min, r.integers(-5, 5, n))
    flag = r.integers(0, 2, n).astype(np.uint8)
    f = np.round(r.normal(size=n), 1)
    text = r.integers(0, len(POOL), n)
    rand = r.permutation(n)
    idx = np.arange(n)
    return {"four": (fixed(INT32, four), INT32, four, None), "days": (fixed(INT32, days), INT32, days, None),
            "low": (fixed(INT64, low, half), INT64, low, half), "flag": (fixed(BOOL, flag, ~half), BOOL, flag, ~half),
            "f": (fixed(FLOAT64, f), FLOAT64, f, None), "text": (utf8_plain([POOL[t] for t in text], four > 0), UTF8, text, four > 0),
            "rand": (fixed(INT64, rand), INT64, rand, None), "idx": (fixed(INT32, idx), INT32, idx, None)}


KEYS = [[("four", True, False)], [("days", False, False)], [("low", True, True)], [("low", False, False)], [("flag", False, True)],
        [("four", False, False), ("f", False, False)], [("low", True, True), ("flag", False, False), ("days", True, True)],
        [("four", True, True), ("text", False, True)], [("flag", True, False), ("text", True, False), ("low", False, True), ("rand", True, False)]]


@pytest.mark.parametrize("n,limit", SIZES)
def test_ties_at_the_limit(ctx, n, limit):
    from minilake_b200.engine import GpuEngine
    cols = _columns(n, n + limit)
    names = list(cols)
    batch = ctx.upload([cols[c][0] for c in names])
    eng = GpuEngine(ctx)

    def topn(keys):
        ctx.profile("topn", reset=True)
        out = eng.topn(batch, batch.types, [SortKey(Col(names.index(c)), cols[c][1], asc=asc, nulls_first=nf) for c, asc, nf in keys], limit)
        took = ctx.profile("topn")[0]
        return eng.fetch(out)[names.index("idx")].values, took

    for keys in KEYS:
        by = []
        for c, asc, nulls_first in reversed(keys):
            _, _, v, valid = cols[c]
            ok = np.ones(n, dtype=bool) if valid is None else valid
            key = np.unique(v, return_inverse=True)[1]
            by += [np.where(ok, key if asc else -key, 0), ok if nulls_first else ~ok]
        rows, took = topn(keys)
        assert np.array_equal(rows, np.lexsort(by)[:limit]), keys
        assert took == 1, keys
    batch.close()
