"""The plans on hit masks (4-clique, annotation of a symmetric relation,
materialized rows): neighbourhoods at the edges of the 32-bit words and of the
32-row blocks, rows of one to many words, up, down and symmetric, in every
layout, batched and in shards, against the oracle; integer work, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(d, density, seed=1):
    """Vertex 0 meets 1..d; among those, each pair with the given density."""
    rng = np.random.default_rng(seed)
    u, v = np.triu_indices(d, 1)
    keep = rng.random(len(u)) < density
    u, v = u[keep] + 1, v[keep] + 1
    u = np.concatenate([np.zeros(d, np.int64), u])
    v = np.concatenate([np.arange(1, d + 1), v])
    return u.astype(np.uint32), v.astype(np.uint32)


def _orient(u, v, kind):
    if kind == "up":
        return u, v
    if kind == "down":
        return v, u
    return np.concatenate([u, v]), np.concatenate([v, u])


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("d,density", [(2, 1.0), (3, 1.0), (31, 1.0), (32, 0.7), (33, 1.0), (34, 0.5), (63, 0.6),
                                       (64, 1.0), (65, 0.9), (97, 0.3), (300, 0.4), (1100, 0.15)])
def test_neighbourhood_sizes(eh, oracle, kind, d, density):
    u, v = _orient(*_graph(d, density), kind)
    o = oracle.Trie(u, v)
    for policy, forced in ((0, 1), (2, 1), (2, 0), (2, 3)):
        t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
        assert t.count("clique4") == o.clique4(), (policy, forced)
        np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
        if d <= 300:
            np.testing.assert_array_equal(t.materialize(), o.triangle_tuples())
        t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
def test_many_neighbourhoods(eh, oracle, kind):
    """R-MAT-12: parts of every size up to a few words, spread ids."""
    u, v = oracle.gen_rmat(3, 12, 16 << 12)
    s, d, n = oracle.preprocess(u, v)
    ids = np.sort(np.random.default_rng(2).choice(1 << 20, n, replace=False)).astype(np.uint32)
    u, v = _orient(ids[s], ids[d], kind)
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v)
    assert t.count("clique4") == o.clique4()
    assert sum(t.count("clique4", shard=(i, 3)) for i in range(3)) == o.clique4()
    assert t.count("clique4", chunk=64, smem_words=64, warps=2) == o.clique4()
    np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
    np.testing.assert_array_equal(t.materialize(), o.triangle_tuples())
    t.free()


def test_batched_cliques(eh, oracle):
    """Graphs of one batch with parts on both sides of 32, an empty one and
    two directions among them."""
    rel = [_orient(*_graph(d, p, seed=d), k) for d, p, k in
           ((5, 1.0, "up"), (40, 0.8, "down"), (33, 1.0, "sym"), (200, 0.3, "up"))]
    rel.insert(2, (np.array([1, 2], np.uint32), np.array([7, 9], np.uint32)))
    want = [oracle.Trie(u, v).clique4() for u, v in rel]
    tries = [eh.Trie(u, v) for u, v in rel]
    b = eh.Batch(tries, "clique4")
    for _ in range(2):
        assert b.run().tolist() == want
    assert eh.count_batched(tries, "clique4").tolist() == want
    b.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("d,extra,core", [(2047, 3000, 0), (2049, 3000, 40), (5000, 20000, 0), (5000, 2000, 300),
                                          (9000, 40000, 120)])
def test_wide_sparse_neighbourhoods(eh, oracle, kind, d, extra, core):
    """Hubs of more than 2048 neighbours (as lowest or highest id) with few
    edges among them, and with a dense core whose rows pass 256 hits."""
    rng = np.random.default_rng(d + core)
    a, b = rng.integers(1, d + 1, extra), rng.integers(1, d + 1, extra)
    ca, cb = np.triu_indices(core, 1)
    ids = np.sort(rng.choice(np.arange(1, d + 1), core, replace=False)) if core else np.zeros(0, np.int64)
    u = np.concatenate([np.zeros(d, np.int64), np.minimum(a, b), ids[ca], np.arange(1, d + 1)])
    v = np.concatenate([np.arange(1, d + 1), np.maximum(a, b), ids[cb], np.full(d, d + 1)])
    keep = u != v
    u, v = _orient(u[keep].astype(np.uint32), v[keep].astype(np.uint32), kind)
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v)
    assert t.count("triangle") == o.triangle()
    assert t.count("clique4") == o.clique4()
    assert eh.count_batched([t, t], "clique4").tolist() == [o.clique4()] * 2
    assert sum(t.count("clique4", shard=(i, 3)) for i in range(3)) == o.clique4()
    np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
    t.free()
