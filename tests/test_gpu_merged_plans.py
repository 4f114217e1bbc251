"""Items that neighbouring entries share, in the plans on hit masks: relations large
enough that entries do share (asserted), against the same plan cut apart and the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("degree", [3, 9])
def test_merged(eh, oracle, kind, degree):
    rng = np.random.default_rng(degree)
    n = 1 << 16
    a, b = rng.integers(0, n, degree * n), rng.integers(0, n, degree * n)
    base = 13 * np.arange(2000)  # small cliques on top, or a sparse relation has none
    ca, cb = np.triu_indices(6, 1)
    a = np.concatenate([a, (base[:, None] + ca).ravel()])
    b = np.concatenate([b, (base[:, None] + cb).ravel()])
    u, v = np.minimum(a, b)[a != b], np.maximum(a, b)[a != b]
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    u, v = u.astype(np.uint32), v.astype(np.uint32)
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v)
    want = dict(triangle=o.triangle(), clique4=o.clique4(), lollipop=o.lollipop())
    assert want["clique4"] > 0
    for query in ("triangle", "clique4") + (("lollipop",) if kind == "sym" else ()):
        got, st = t.count(query, stats=True)
        own, ost = t.count(query, stats=True, record=True)
        assert got == own == want[query], query
        assert st["work_items"] < 0.7 * ost["work_items"], query
    assert t.count("lollipop") == want["lollipop"]
    np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
    np.testing.assert_array_equal(t.materialize(), o.triangle_tuples())
    t.free()
