"""4-cliques on hit masks where there are fewer units than warps: a unit's blocks are
shared by up to eight warps; one wide part or several, alone, in a batch and in shares;
against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(d, density, hubs, kind):
    rng = np.random.default_rng(d + hubs)
    x = hubs + np.arange(d)
    m = int(density * d)
    a, b = rng.integers(0, d, m), rng.integers(0, d, m)
    u = np.concatenate([np.repeat(np.arange(hubs), d), np.zeros(hubs - 1, np.int64), hubs + np.minimum(a, b)])
    v = np.concatenate([np.tile(x, hubs), np.arange(1, hubs), hubs + np.maximum(a, b)])
    k = min(d, 36)
    ca, cb = np.triu_indices(k, 1)  # a clique among the last ones
    u, v = np.concatenate([u, hubs + d - k + ca]), np.concatenate([v, hubs + d - k + cb])
    u, v = u[u != v], v[u != v]
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u.astype(np.uint32), v.astype(np.uint32)


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("hubs", [1, 4])
@pytest.mark.parametrize("d", [33, 40, 63, 64, 65, 256, 300, 1000, 2047, 2049, 5000])
def test_clique(eh, oracle, d, hubs, kind):
    tries, want = [], []
    for density in (1, 20):
        u, v = _relation(d, density, hubs, kind)
        want.append(oracle.Trie(u, v).clique4())
        tries.append(eh.Trie(u, v))
        assert tries[-1].count("clique4") == want[-1]
        for world in (2, 3):
            assert sum(tries[-1].count("clique4", shard=(r, world)) for r in range(world)) == want[-1]
    b = eh.Batch(tries, "clique4")
    for _ in range(2):
        assert b.run().tolist() == want
    b.free()
    for t in tries:
        t.free()
