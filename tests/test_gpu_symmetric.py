"""Symmetric relations stage only the part of N(b) above b.  The plans over
relations where that part is empty, short, split inside a bitset word, longer
than a warp's and than a block's staging region (a hub with the smallest id),
or the whole set, against the oracle; integer work, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(kind):
    rng = np.random.default_rng(len(kind))
    if kind == "hub_low":  # id 0 meets everyone: its part is the whole set
        n, m = 9000, 20000
        u = np.concatenate([np.zeros(n - 1, np.int64), rng.integers(0, n, m)])
        v = np.concatenate([np.arange(1, n), rng.integers(0, n, m)])
    elif kind == "hub_high":  # the largest id meets everyone: its part is empty
        n, m = 9000, 20000
        u = np.concatenate([np.full(n - 1, n - 1), rng.integers(0, n, m)])
        v = np.concatenate([np.arange(0, n - 1), rng.integers(0, n, m)])
    elif kind == "dense":  # every set crosses its own id inside a word
        n, m = 300, 20000
        u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    else:  # sparse wide ids
        ids = np.sort(rng.choice(1 << 22, 400, replace=False))
        u, v = ids[rng.integers(0, 400, 6000)], ids[rng.integers(0, 400, 6000)]
    keep = u != v
    u, v = u[keep].astype(np.uint32), v[keep].astype(np.uint32)
    return np.concatenate([u, v]), np.concatenate([v, u])


@pytest.mark.parametrize("kind", ["hub_low", "hub_high", "dense", "wide"])
@pytest.mark.parametrize("policy,forced", [(0, 1), (2, 1), (2, 0), (2, 3)])
def test_symmetric_plans(eh, oracle, kind, policy, forced):
    u, v = _relation(kind)
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
    assert t.count("triangle") == o.triangle()
    assert t.count("triangle", smem_words=64, warps=2) == o.triangle()
    assert t.count("clique4") == o.clique4()
    np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
    assert t.count("lollipop") == o.lollipop()
    assert t.count("barbell") == o.barbell()
    t.free()
