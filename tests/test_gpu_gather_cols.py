"""ORDER BY results gathered from several columns at once: widths 1, 4 and 8 with and without validity, more
columns than a launch takes, columns that share a launch and ones too large to, row counts about a
warp's validity word and a thread's batch of rows.  The permutation is known, so values and validity are
compared exactly."""
import numpy as np
import pytest

from minilake_b200.abi import BOOL, DATE, FLOAT64, INT32, INT64, Col, SortKey
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu

KINDS = [(INT64, np.int64), (FLOAT64, np.float64), (INT32, np.int32), (DATE, np.int32), (BOOL, np.uint8)]


@pytest.mark.parametrize("n,ncols", [(1025, 3), (1056, 19), (4095, 1), (4097, 17), (100_003, 5), (3_000_001, 4), (9_000_000, 2)])
@pytest.mark.parametrize("nulls", [False, True])
def test_columns_follow_the_order(n, ncols, nulls):
    from minilake_b200 import gpu
    from minilake_b200.engine import GpuEngine
    r = np.random.default_rng(n + ncols)
    perm = r.permutation(n)
    cols, want = [fixed(INT64, perm.astype(np.int64))], []
    back = np.argsort(perm)
    for c in range(ncols):
        t, dt = KINDS[c % len(KINDS)]
        v = r.integers(0, 2 if t == BOOL else 1 << 30, n).astype(dt)
        mask = r.random(n) > 0.25 if nulls and c % 3 != 2 else None
        cols.append(fixed(t, v, mask))
        want.append((v[back], None if mask is None else mask[back]))
    ctx = gpu.Context(0)
    engine = GpuEngine(ctx)
    batch = ctx.upload(cols)
    got = engine.fetch(engine.topn([batch], batch.types, [SortKey(Col(0), INT64)], None))
    assert np.array_equal(got[0].values, np.arange(n))
    for g, (v, mask) in zip(got[1:], want):
        if mask is None:
            assert g.validity is None or g.valid_mask().all()
            assert np.array_equal(g.values, v)
        else:
            assert np.array_equal(g.valid_mask(), mask)
            assert np.array_equal(g.values[mask], v[mask])
    ctx.close()
