"""Neighbouring entries that share a work item: relations of many small sets
whose groups of 16 or 8 entries lie around the limits (128 rows, 1024 candidates
and elements), entries without rows among them, one long row in a group, in
every direction, in shards and batched; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(per, kind, seed):
    """Around `per` rows end at each entry; sparse ids; a few sets of hundreds."""
    rng = np.random.default_rng(seed)
    n = 24000 if per == 8 else 2600
    u = rng.integers(0, n, per * n)
    v = rng.integers(0, n, per * n)
    hub = rng.integers(0, 40)
    u = np.concatenate([u, np.full(500, hub)])
    v = np.concatenate([v, rng.choice(n, 500, replace=False)])
    ids = np.sort(rng.choice(5 * n, n, replace=False)).astype(np.uint32)
    u, v = ids[u], ids[v]
    if kind != "general":
        keep = u != v
        u, v = np.minimum(u, v)[keep], np.maximum(u, v)[keep]
        if kind == "down":
            u, v = v, u
        if kind == "sym":
            u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u, v


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general"])
@pytest.mark.parametrize("per", [1, 2, 7, 8, 9, 16, 17, 24])
def test_shared_items(eh, oracle, kind, per):
    for seed in (per, per + 100):
        u, v = _relation(per, kind, seed)
        o = oracle.Trie(u, v)
        t = eh.Trie(u, v)
        # entries share items past four of them per resident warp: the default
        # schedule reaches that with 24,000 entries, large staging with 2,600
        kw = dict() if per == 8 else dict(smem_words=16384, warps=1)
        assert t.count("triangle", **kw) == o.triangle()
        assert sum(t.count("triangle", shard=(i, 3), **kw) for i in range(3)) == o.triangle()
        assert t.count("triangle", record=True) == o.triangle()
        assert t.count("clique4", **kw) == o.clique4()
        assert sum(t.count("clique4", shard=(i, 3), **kw) for i in range(3)) == o.clique4()
        np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
        np.testing.assert_array_equal(t.materialize(), o.triangle_tuples())
        for q, want in (("triangle", o.triangle()), ("clique4", o.clique4())):
            b = eh.Batch([t, t], q, config=kw)
            assert b.run().tolist() == [want, want]
            b.free()
        t.free()
