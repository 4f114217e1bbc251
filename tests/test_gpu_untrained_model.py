"""A cost model that predicts nothing (fresh weights, or trained on something else) lays
a trie out and cuts its work: counts stay exact and no item outgrows four chunks of
work, whatever it predicts of a hub."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROW_COST = 8


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("seed", [1, 4, 6])
def test_items_are_bounded(eh, ctx, oracle, symmetric, seed):
    u, v = eh.gen_chunglu(5, 1 << 16, 16 << 16, 2.1, ctx=ctx)
    s, d, _ = eh.preprocess(u, v, symmetric=symmetric, ctx=ctx)
    t = eh.Trie(s, d, ctx=ctx)
    want = {q: t.count(q) for q in ("triangle", "lollipop")}
    assert want["triangle"] == oracle.Trie(s.numpy(), d.numpy()).triangle()
    longest = t.info()["max_set"]
    m = eh.Model([6, 32, 32, 1], seed=seed, ctx=ctx)
    t.relayout(policy=eh.LEARNED, model=m)
    for chunk in (4096, 20_000):
        for query in want:
            got, st = t.count(query, chunk=chunk, stats=True, block_items=False, record=True)
            assert got == want[query]
            rec = eh.timing_records(ctx)
            assert len(rec) == st["work_items"]
            # an item ends with the row that reaches its share
            assert rec[:, 1].max() <= 2 * 4 * chunk + longest, (chunk, query)
        assert t.count("triangle", chunk=chunk) == want["triangle"]
        assert sum(t.count("triangle", chunk=chunk, shard=(r, 3)) for r in range(3)) == want["triangle"]
    m.free()
    t.free()
