"""4-cliques of parts of more than 2048 neighbours: units shared by a block, by the
words of nearly empty rows or by all blocks of words, and units large enough for the
list that all blocks work off; alone, in a batch, in shares; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(d, subs, share, rows, kind):
    """A hub next to d, the first `subs` of them next to a share of the rest, and rows
    among the rest; a clique at the end."""
    rng = np.random.default_rng(d + subs)
    u, v = [np.zeros(d, np.int64)], [1 + np.arange(d)]
    for k in range(subs):
        x = 1 + subs + np.flatnonzero(rng.random(d - subs) < share)
        x = np.concatenate([np.arange(k + 2, subs + 1), x])
        u.append(np.full(len(x), k + 1))
        v.append(x)
    a, b = 1 + rng.integers(0, d, rows), 1 + rng.integers(0, d, rows)
    ca, cb = np.triu_indices(30, 1)
    u, v = np.concatenate(u + [np.minimum(a, b), d - 30 + ca]), np.concatenate(v + [np.maximum(a, b), d - 30 + cb])
    u, v = u[u != v], v[u != v]
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u.astype(np.uint32), v.astype(np.uint32)


CASES = [
    (2049, 10, 0.5, 4000),     # a block's warps, dense
    (2100, 10, 0.005, 4000),   # and by rows' words
    (4096, 40, 0.3, 9000),
    (6500, 24, 0.5, 20_000),   # past the list's limit, dense
    (8200, 9, 0.03, 60_000),
    (30_000, 12, 0.0135, 60_000),  # past it by words, more of a row than are held at a time
    (30_000, 12, 0.02, 60_000),    # and just not by words
    (30_000, 8, 0.2, 20_000),
]


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("case", CASES)
def test_clique(eh, oracle, case, kind):
    u, v = _relation(*case, kind)
    want = oracle.Trie(u, v).clique4()
    assert want > 0
    t = eh.Trie(u, v)
    for _ in range(2):
        assert t.count("clique4") == want
    for world in (2, 3):
        assert sum(t.count("clique4", shard=(r, world)) for r in range(world)) == want
    small = eh.Trie(*(np.asarray(x, np.uint32) for x in np.triu_indices(40, 1)))
    b = eh.Batch([small, t, t], "clique4")
    for _ in range(3):
        assert b.run().tolist() == [91390, want, want]
    b.free()
    t.free()
    small.free()
