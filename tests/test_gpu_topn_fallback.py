"""ORDER BY ... LIMIT where the selection gives up (more equal rows at the limit than it sorts, told apart
only past a string's first eight bytes) and another route answers: rows that are not the result may not be
charged to a budget, and a long string among them may not end the call.  The rows kept are a stable sort's."""
import numpy as np
import pytest

from minilake_b200.abi import FLOAT64, INT32, UTF8, Col, SortKey
from minilake_b200.columns import fixed, utf8_plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1000, 2048])
@pytest.mark.parametrize("first,budget", [(3_000_000, 0), (200_000, 96 << 20)])
def test_a_long_string_among_the_rows_that_are_not_the_result(limit, first, budget):
    from minilake_b200.engine import GpuEngine
    from minilake_b200.gpu import Context
    n = 70_001
    r = np.random.default_rng(limit)
    key = r.integers(0, 4, n)
    key[0] = 3
    tail = r.integers(0, 10_000, n)
    names = [b"Customer#%05d" % t for t in tail]
    names[0] = b"x" * first
    ctx = Context(0, hbm_budget=budget)
    batch = ctx.upload([fixed(INT32, key), utf8_plain(names), fixed(FLOAT64, np.arange(n))])
    keys = [SortKey(Col(0), INT32, asc=True), SortKey(Col(1), UTF8, asc=False)]
    eng = GpuEngine(ctx)
    out = eng.fetch(eng.topn(batch, [INT32, UTF8, FLOAT64], keys, limit))
    order = np.lexsort([-tail, key])  # row 0 is not among the first: its key is the last one
    assert key[order[limit - 1]] == 0
    want = order[:limit]
    assert np.array_equal(out[2].values, want)
    assert out[1].strings() == [names[i] for i in want]
    ctx.close()
