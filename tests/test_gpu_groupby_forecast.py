"""GROUP BY without a size hint, small batches and then a large one: the table is sized for the groups the
large batch's rows bring, not as if its first rows had brought the earlier ones too.  A table for G groups has
2 G slots at least, rounded up to a power of two; a forecast of up to twice the groups stays below 8 G."""
import numpy as np
import pytest

from minilake_b200.abi import COUNT_STAR, INT64, SUM, AggSpec, Col
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small,new", [(100_000, 0), (100_000, 100_000), (30_000, 0), (30_000, 900_000)])
def test_small_batches_before_a_large_one(small, new):
    from minilake_b200.gpu import Context, HashAggregateSink
    ctx = Context(0)
    r = np.random.default_rng(new)
    m, n = 10 * small, 10_000_000
    first, second = r.permutation(m), r.integers(0, m + new, n)
    sink = HashAggregateSink(ctx, [INT64], [(Col(0), INT64)], [AggSpec(COUNT_STAR), AggSpec(SUM, Col(0), INT64)])
    local = sink.create_local()
    for part in np.split(first, 10) + [second]:
        batch = ctx.upload([fixed(INT64, part * 7 - 3)])
        local.sink(batch)
        batch.close()
    local.combine()
    stats = sink.stats()
    out = sink.finalize().fetch()
    count = np.bincount(first, minlength=m + new) + np.bincount(second, minlength=m + new)
    key = (out[0].values + 3) // 7
    assert np.array_equal(np.sort(key), np.flatnonzero(count))
    assert np.array_equal(out[1].values, count[key]) and np.array_equal(out[2].values, count[key] * out[0].values)
    assert stats["groups"] == len(key)
    assert stats["capacity"] <= 8 * len(key)
    sink.close()
    ctx.close()
