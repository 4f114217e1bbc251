"""Annotation on hit masks where parts are wide: units shared by the warps of a block
from 4097 elements on, by up to eight warps; several wide parts, and narrow ones beside
them; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(d, rows, hubs, top):
    rng = np.random.default_rng(d + rows)
    u, v = [], []
    for h in range(hubs):
        x = hubs + np.arange(d if h == 0 else d - 7 * h)
        u.append(np.full(len(x), h))
        v.append(x)
    a, b = hubs + rng.integers(0, d, rows), hubs + rng.integers(0, d, rows)
    k = min(d, 40)
    ca, cb = np.triu_indices(k, 1)  # a dense corner
    u, v = np.concatenate(u + [a, hubs + ca]), np.concatenate(v + [b, hubs + d - k + cb])
    u, v = u[u != v], v[u != v]
    if top:  # the hubs are the last ids: their parts are empty, the leaves' short
        u, v = d + hubs - u, d + hubs - v
    return np.concatenate([u, v]).astype(np.uint32), np.concatenate([v, u]).astype(np.uint32)


@pytest.mark.parametrize("top", [False, True])
@pytest.mark.parametrize("hubs", [1, 3])
@pytest.mark.parametrize("d", [31, 32, 33, 1000, 2048, 4095, 4096, 4097, 4128, 8191, 8193, 16383, 20000])
def test_annotation(eh, oracle, d, hubs, top):
    for rows in (50, 8 * d):
        u, v = _relation(d, rows, hubs, top)
        o = oracle.Trie(u, v)
        t = eh.Trie(u, v)
        np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
        assert t.count("lollipop") == o.lollipop()
        t.free()


def test_many_wide_parts(eh, oracle):
    """A hundred hubs, so that blocks find several wide units in one look."""
    rng = np.random.default_rng(1)
    hubs, d = 100, 6000
    m = rng.random((hubs, d)) < 0.8
    h, x = np.nonzero(m)
    a, b = hubs + rng.integers(0, d, 9_000), hubs + rng.integers(0, d, 9_000)
    u, v = np.concatenate([h, a]), np.concatenate([x + hubs, b])
    u, v = u[u != v], v[u != v]
    u, v = np.concatenate([u, v]).astype(np.uint32), np.concatenate([v, u]).astype(np.uint32)
    o = oracle.Trie(u, v)
    t = eh.Trie(u, v)
    np.testing.assert_array_equal(t.triangle_annotation(), o.triangle_per_vertex())
    assert t.count("barbell") == o.barbell()
    t.free()
