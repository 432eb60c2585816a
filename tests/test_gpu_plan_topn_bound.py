"""Replayed plans whose top-N runs over a large group table behind a bound on the first key: the replay has
to give the planning run's rows and order (that run orders all groups), for every aggregate as the first
key, ascending and descending, limits up to the warp lists' 32, values that tie in all groups, NaN and
negative values, and after the data changed in place; too few groups make the plan stale.  Doubles are
whole numbers, so sums are exact in any order."""
import numpy as np
import pytest

from minilake_b200.abi import (AVG, COUNT, COUNT_STAR, FLOAT64, INT32, INT64, MAX, MIN, SUM, AggSpec, Col, Probe, SortKey)

from test_gpu_query import _torch_table

pytestmark = pytest.mark.gpu

ND, NF = 60_000, 400_000
AGGS = [AggSpec(SUM, Col(1), FLOAT64), AggSpec(COUNT_STAR), AggSpec(AVG, Col(1), FLOAT64), AggSpec(MIN, Col(1), FLOAT64),
        AggSpec(MAX, Col(2), INT32), AggSpec(SUM, Col(2), INT64), AggSpec(COUNT, Col(1), FLOAT64)]
TYPES = [FLOAT64, INT64, FLOAT64, FLOAT64, INT32, INT64, INT64]


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200.gpu import Context
    c = Context(0)
    yield c
    c.close()


def _same(got, want):
    for g, w in zip(got, want):
        assert g.values.dtype == w.values.dtype and g.values.tobytes() == w.values.tobytes()


@pytest.mark.parametrize("limit", [1, 10, 32])
@pytest.mark.parametrize("first", range(len(AGGS)))
@pytest.mark.parametrize("asc", [False, True])
def test_replay_gives_the_planning_runs_rows(ctx, first, asc, limit):
    import torch
    from minilake_b200.gpu import HashAggregateSink, JoinBuildSink, Query, StalePlan
    rng = np.random.default_rng(first * 10 + limit)
    key = rng.permutation(ND).astype(np.int64) + 11
    fk = key[rng.integers(0, ND, NF)]
    v = rng.integers(-1000, 1000, NF).astype(np.float64)
    i = rng.integers(-(1 << 30), 1 << 30, NF, dtype=np.int32)
    dim, _ = _torch_table([(INT64, key)])
    fact, t = _torch_table([(INT64, fk), (FLOAT64, v), (INT32, i)])
    keys = [SortKey(Col(1 + first), TYPES[first], asc=asc), SortKey(Col(0), INT64)]
    if limit == 1:
        keys = keys[:1]  # ties keep the groups' order

    def planned():
        q = Query(ctx)
        jt = q.add_build(JoinBuildSink(ctx, [INT64], [(Col(0), INT64)]), dim.ml)
        q.set_aggregate(HashAggregateSink(ctx, [INT64, FLOAT64, INT32], [(Col(0), INT64)], AGGS, [Probe(jt, [(Col(0), INT64)])]), fact.ml)
        q.set_topn(keys, limit)
        return q, q.run().fetch()

    q, want = planned()
    assert len(want[0]) == limit
    for _ in range(2):
        _same(q.run().fetch(), want)
    assert q.stats()["why_not"] == "" and q.stats()["replays"] == 2
    data = {"ties": np.full(NF, 7.0), "nan": np.where(rng.random(NF) < 0.001, np.nan, v), "zero": np.where(rng.random(NF) < 0.5, -0.0, 0.0),
            "inf": np.where(rng.random(NF) < 0.001, np.inf, -v)}
    for name, x in data.items():
        t[1].copy_(torch.from_numpy(x))
        got = q.run().fetch()
        q2, want2 = planned()
        _same(got, want2)
        q2.close()
    t[0].fill_(int(key[0]))  # one group is left
    if limit > 1:
        with pytest.raises(StalePlan):
            q.run()
    else:
        assert q.run().fetch()[0].values[0] == key[0]
    q.close()
