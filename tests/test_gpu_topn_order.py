"""ORDER BY ... LIMIT over columns in an order that a sample could miss (sorted, reversed, sorted runs), at
the row counts of both sample sizes: the rows kept are a stable sort's, and the selection finds them (as many
launches as for random values; another route takes more)."""
import numpy as np
import pytest

from minilake_b200.abi import FLOAT64, INT32, Col, SortKey
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield ctx
    ctx.close()


def _topn(ctx, v, limit, asc):
    from minilake_b200.engine import GpuEngine
    batch = ctx.upload([fixed(FLOAT64, v), fixed(INT32, np.arange(len(v)))])
    eng = GpuEngine(ctx)
    before = ctx.kernel_launches()
    out = eng.topn(batch, batch.types, [SortKey(Col(0), FLOAT64, asc=asc)], limit)
    launches = ctx.kernel_launches() - before
    rows = eng.fetch(out)[1].values
    batch.close()
    return rows, launches


@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("n,limit", [(2_500_003, 10), (4 << 20, 32), (4_500_001, 100), (9_000_007, 10), (300_001, 2000)])
def test_ordered_columns(ctx, n, limit, asc):
    rand = np.random.default_rng(n).random(n)
    _, launches = _topn(ctx, rand, limit, asc)
    up = np.sort(rand)
    m = n // 32 * 32
    runs = np.concatenate([np.sort(rand[:m].reshape(32, -1), axis=1).ravel(), rand[m:]])
    for v in (up, up[::-1].copy(), runs, np.roll(up, n // 3)):
        rows, took = _topn(ctx, v, limit, asc)
        assert np.array_equal(rows, np.argsort(v if asc else -v, kind="stable")[:limit])
        assert took == launches
