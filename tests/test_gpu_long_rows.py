"""Rows of many candidates, as relations have them whose hubs are among the low ids
(a program's own ids, no degree order): items of a block with any number of rows, in
batches of 1 to 32, and rows the warp runs along; against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIRST, HUBS, POOL = 1000, 4, 24000


def _relation(sources, kind):
    """`sources` vertices, each next to most of a pool and to HUBS hubs, which are next
    to a few thousand of the pool: sets for a block's staging, one long row per source."""
    rng = np.random.default_rng(sources)
    hubs = FIRST - HUBS + np.arange(HUBS)
    u, v = [], []
    for a in range(sources):
        x = np.concatenate([hubs, FIRST + np.flatnonzero(rng.random(POOL) < 0.9)])
        u.append(np.full(len(x), a))
        v.append(x)
    for b in hubs:
        x = FIRST + np.flatnonzero(rng.random(POOL) < 0.2)
        u.append(np.full(len(x), b))
        v.append(x)
    u, v = np.concatenate(u), np.concatenate(v)
    if kind == "down":
        u, v = FIRST + POOL - u, FIRST + POOL - v
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    if kind == "general":
        u, v = np.concatenate([u, v[::5], u[:3]]), np.concatenate([v, u[::5], u[:3]])
    return u.astype(np.uint32), v.astype(np.uint32)


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general"])
@pytest.mark.parametrize("sources", [9, 31, 33, 65, 127, 129])
def test_block_items_of_few_rows(eh, oracle, kind, sources):
    u, v = _relation(sources, kind)
    want = oracle.Trie(u, v).triangle()
    assert want > 0
    for policy, forced in ((0, 1), (2, 0), (2, 1)):
        t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
        for warps in (2, 7, 8, 16):
            assert t.count("triangle", chunk=1 << 20, warps=warps) == want, (policy, forced, warps)
            assert t.count("triangle", chunk=1 << 20, warps=warps, block_items=False) == want
        assert sum(t.count("triangle", chunk=1 << 16, shard=(r, 3)) for r in range(3)) == want
        t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general"])
@pytest.mark.parametrize("n", [255, 256, 257, 287, 288, 289, 479, 480, 481, 511, 512, 513, 768, 1000])
def test_row_lengths(eh, oracle, kind, n):
    """Rows of n candidates and one more or less, among short ones, in every way a set
    is staged."""
    rng = np.random.default_rng(n)
    first, last = 100, 100 + n + 40
    u, v = [], []
    for a in range(40):  # b = 50 .. 54, then exactly n - 1, n or n + 1 candidates, or a few
        size = (n - 1, n, n + 1, 3)[a % 4]
        x = np.concatenate([50 + np.arange(5), first + np.sort(rng.permutation(last - first)[:size])])
        u.append(np.full(len(x), a))
        v.append(x)
    for b in range(50, 55):
        x = first + np.flatnonzero(rng.random(last - first) < 0.3)
        u.append(np.full(len(x), b))
        v.append(x)
    u, v = np.concatenate(u), np.concatenate(v)
    if kind == "down":
        u, v = last - u, last - v
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    if kind == "general":
        u, v = np.concatenate([u, v[::7], u[:3]]), np.concatenate([v, u[::7], u[:3]])
    u, v = u.astype(np.uint32), v.astype(np.uint32)
    want = oracle.Trie(u, v).triangle()
    for policy, forced in ((0, 1), (2, 0), (2, 1), (2, 3)):
        t = eh.Trie(u, v, policy=policy, forced=forced, max_bitset_bytes=1 << 40)
        assert t.count("triangle") == want, (policy, forced)
        assert t.count("triangle", smem_words=64) == want
        assert t.count("triangle", long_row=1000, chunk=700) == want
        assert eh.count_batched([t, t], "triangle").tolist() == [want, want]
        t.free()
