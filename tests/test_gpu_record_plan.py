"""Timing records are taken on the items that the query runs without them (where
entries share none): the cost model learns what its layouts will cost."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(n, m, kind):
    """A hub next to all and a few rows: fewer entries than warps, none shared."""
    rng = np.random.default_rng(n)
    a, b = rng.integers(1, n, m), rng.integers(1, n, m)
    u = np.concatenate([np.zeros(n - 1, np.int64), np.minimum(a, b)])
    v = np.concatenate([np.arange(1, n), np.maximum(a, b)])
    u, v = u[u != v].astype(np.uint32), v[u != v].astype(np.uint32)
    if kind == "sym":
        return np.concatenate([u, v]), np.concatenate([v, u])
    return u, v


@pytest.mark.parametrize("kind", ["up", "sym"])
@pytest.mark.parametrize("query", ["triangle", "clique4", "lollipop"])
@pytest.mark.parametrize("n,m", [(50, 100), (4000, 3000), (60_000, 3000), (1_000_000, 3000)])
def test_records_of_the_plan(eh, ctx, n, m, query, kind):
    t = eh.Trie(*_relation(n, m, kind), ctx=ctx)
    want, st = t.count(query, stats=True)
    got, rst = t.count(query, stats=True, record=True)
    assert got == want
    assert rst["work_items"] == st["work_items"]
    rec = eh.timing_records(ctx)
    assert len(rec) == st["work_items"]
    assert rec[:, 1].astype(np.float64).sum() == pytest.approx(st["wedges"], rel=1e-4)
    t.free()
