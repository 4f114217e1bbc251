"""The four ways a row is counted (word trips, flattened words, element trips,
flattened elements) around their boundaries: common ranges of 1 to 70 words at
several alignments, candidate runs around long_row and 32, staged in a warp's
region or read from global memory, up, down, symmetric and general; against the
oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relation(words, kind, density, offset):
    """A few low vertices, each meeting most of a range of `words` words (and
    each other), and some of the range's vertices meeting a few more."""
    rng = np.random.default_rng(words * 7 + offset)
    n = 6
    first = 64 + offset
    span = np.arange(first, first + 64 * words - offset)
    u, v = [], []
    for a in range(n):
        x = span[rng.random(len(span)) < density]
        x = np.concatenate([np.arange(a + 1, n), x])
        u.append(np.full(len(x), a))
        v.append(x)
    for a in span[:: max(1, len(span) // 40)]:
        x = np.unique(rng.integers(a + 1, first + 64 * words + 50, 45))
        u.append(np.full(len(x), a))
        v.append(x)
    u, v = np.concatenate(u).astype(np.uint32), np.concatenate(v).astype(np.uint32)
    if kind == "down":
        return v, u
    if kind == "sym":
        return np.concatenate([u, v]), np.concatenate([v, u])
    if kind == "general":
        return np.concatenate([u, v[::3], u[:5]]), np.concatenate([v, u[::3], u[:5]])
    return u, v


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general"])
@pytest.mark.parametrize("words", [1, 2, 15, 16, 17, 31, 32, 33, 64, 70])
def test_row_classes(eh, oracle, kind, words):
    for density, offset in ((0.9, 0), (0.3, 37), (0.05, 63)):
        u, v = _relation(words, kind, density, offset)
        want = oracle.Trie(u, v).triangle()
        for policy, forced in ((0, 1), (2, 0), (2, 1), (2, 3)):
            t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
            assert t.count("triangle") == want, (density, policy, forced)
            assert t.count("triangle", long_row=1, chunk=100) == want
            assert t.count("triangle", long_row=1000, smem_words=64, warps=1) == want
            assert eh.count_batched([t, t], "triangle").tolist() == [want, want]
            t.free()
