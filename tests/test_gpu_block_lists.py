"""Plans on hit masks over block bitsets: a set that fits the warp's shared memory is
staged by its elements, a larger one probed where it lies; sizes around the limit;
against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("size", [60, 63, 64, 65, 70, 400, 1279, 1280, 1281, 1400])
def test_block_sets(eh, oracle, size, kind):
    rng = np.random.default_rng(size)
    n, far = 24, 40 + 9 * np.arange(1600)
    u, v = [np.repeat(np.arange(n), n)], [np.tile(np.arange(n), n)]
    for a in range(n):
        x = far[np.sort(rng.permutation(len(far))[: size + a % 3 - 1])]
        u.append(np.full(len(x), a))
        v.append(x)
    a, b = far[rng.integers(0, len(far), 4000)], far[rng.integers(0, len(far), 4000)]
    u, v = np.concatenate(u + [np.minimum(a, b)]), np.concatenate(v + [np.maximum(a, b)])
    u, v = u[u < v].astype(np.uint32), v[u < v].astype(np.uint32)
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v, policy=eh.FORCED, forced=eh.BLOCK_BITSET)
    clique, lollipop = o.clique4(), o.lollipop()
    for kw in (dict(), dict(smem_words=64), dict(chunk=60)):
        assert t.count("clique4", **kw) == clique, kw
        assert t.count("lollipop", **kw) == lollipop, kw
    if kind != "sym":
        np.testing.assert_array_equal(t.materialize(), o.triangle_tuples())
    t.free()
