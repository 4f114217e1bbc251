"""The annotated triangle pass of relations that run it without hit masks (up, down,
general): sets staged as a list, a plain bitmap or a compressed one, by their span and
the shared memory there is; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(span, kind):
    """100 low vertices next to most of each other and to a few hundred of `span` ids,
    of which some meet a few more."""
    rng = np.random.default_rng(span)
    n = 100
    far = n + np.unique(rng.integers(0, span, 400))
    u, v = [np.repeat(np.arange(n), n)], [np.tile(np.arange(n), n)]
    for a in range(n):
        x = far[rng.random(len(far)) < rng.random()]
        u.append(np.full(len(x), a))
        v.append(x)
    for a in far[::9]:
        x = far[far > a][:30]
        u.append(np.full(len(x), a))
        v.append(x)
    u, v = np.concatenate(u), np.concatenate(v)
    u, v = u[u < v], v[u < v]
    if kind == "down":
        u, v = v, u
    if kind == "general":
        u, v = np.concatenate([u, v[::3], u[:5]]), np.concatenate([v, u[::3], u[:5]])
    return u.astype(np.uint32), v.astype(np.uint32)


@pytest.mark.parametrize("kind", ["up", "down", "general"])
@pytest.mark.parametrize("span", [401, 3000, 20_000, 200_000, 40_000_000])
def test_annotation(eh, oracle, kind, span):
    u, v = _relation(span, kind)
    o = oracle.Trie(u, v)
    per, lollipop, barbell = o.triangle_per_vertex(), o.lollipop(), o.barbell()
    for policy, forced in ((0, 1), (2, 0), (2, 1), (2, 3)):
        if span > 1 << 20 and (policy, forced) == (2, 0):
            continue  # bitsets of the whole span for every set
        t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
        np.testing.assert_array_equal(t.triangle_annotation(), per)
        for kw in (dict(), dict(chunk=1 << 20), dict(smem_words=64), dict(smem_words=400, warps=3), dict(chunk=50), dict(long_row=1)):
            assert t.count("lollipop", **kw) == lollipop, (policy, forced, kw)
        assert t.count("barbell") == barbell
        t.free()
