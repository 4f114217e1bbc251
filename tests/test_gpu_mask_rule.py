"""Which relations run on hit masks.  Without rows that have candidates nothing but
the plan's bookkeeping runs.  Small neighbourhoods (up to 32 elements: a row per
lane) around that line, few of them and more than there are warps for one at a
time, in shares and batches; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _orient(u, v, kind):
    if kind == "down":
        return v, u
    if kind == "sym":
        return np.concatenate([u, v]), np.concatenate([v, u])
    return u, v


def _launches(t, query):
    return t.count(query, stats=True)[1]["launches"]


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
def test_no_candidates(eh, kind):
    n = 5000
    star = np.zeros(n, np.uint32), np.arange(1, n + 1, dtype=np.uint32)
    path = np.arange(n, dtype=np.uint32), np.arange(1, n + 1, dtype=np.uint32)
    for u, v in (star, path):
        if kind == "down":  # the star's centre as the highest id: its rows have no candidates either
            u, v = n - u, n - v
        t = eh.Trie(*_orient(u, v, "sym" if kind == "sym" else "up"))
        if t.count("triangle", stats=True)[1]["wedges"] == 0:
            for q in ("clique4", "lollipop"):
                assert t.count(q) == 0
                # no plan, no masks: the root bag's launch alone
                assert _launches(t, q) == (1 if q == "lollipop" else 0)
        assert t.count("clique4", shard=(1, 3)) == 0
        assert len(t.materialize()) == 0
        t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("n", [4, 32, 33, 34, 35])
def test_small_sets(eh, oracle, kind, n):
    u, v = np.triu_indices(n, 1)
    u, v = _orient(u.astype(np.uint32), v.astype(np.uint32), kind)
    want = oracle.Trie(u, v).clique4()
    t = eh.Trie(u, v)
    assert t.count("clique4") == want
    assert sum(t.count("clique4", shard=(r, 3)) for r in range(3)) == want
    b = eh.Batch([t] * 5, "clique4")
    assert b.run().tolist() == [want] * 5
    b.free()
    t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
def test_many_small_neighbourhoods(eh, oracle, kind):
    """Groups of five vertices, a 4-clique's neighbourhoods among them: up to 4,
    and more than 8 head entries for each warp of the device."""
    a, b = np.triu_indices(5, 1)
    for groups in (1, 3, 2_000, 40_000):
        base = 5 * np.arange(groups)[:, None]
        u, v = (base + a).ravel().astype(np.uint32), (base + b).ravel().astype(np.uint32)
        u, v = _orient(u, v, kind)
        want = oracle.Trie(u, v).clique4()
        assert want == groups * 5 * (24 if kind == "sym" else 1)
        t = eh.Trie(u, v)
        assert t.count("clique4") == want
        assert sum(t.count("clique4", shard=(r, 4)) for r in range(4)) == want
        t.free()
