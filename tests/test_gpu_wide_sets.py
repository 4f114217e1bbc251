"""Bitset structures of sets that are wide, or long, or both: around the sizes where
a warp, a block and the grid build them (2048 and 131,072 elements or words; few
elements over up to 2^22 words stay with the blocks).  Every set's reference-format bytes
equal the same set's built alone from the elements on the CPU, and many wide, thin
sets cost a small share of one grid-wide pass each."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RANGE, UINT, BLOCK = 0, 1, 3


def _elements(n, words, seed):
    """n ascending values over a span of exactly `words` 64-bit words."""
    rng = np.random.default_rng(seed)
    base = 64 * int(rng.integers(1, 1000)) + 5
    last = ((base >> 6) + words - 1) * 64 + 63
    inner = rng.integers(base + 1, last, 2 * n)
    v = np.unique(np.concatenate([[base, last], inner]))
    if len(v) > n:
        keep = np.sort(rng.choice(len(v) - 2, n - 2, replace=False)) + 1
        v = np.concatenate([[v[0]], v[keep], [v[-1]]])
    return v.astype(np.uint32)


@pytest.mark.parametrize("layout", [RANGE, BLOCK])
def test_sets_of_every_builder(eh, layout):
    sizes = [(2, 1), (3, 2049), (300, 131_072), (300, 131_073), (300, 600_000), (2047, 40), (2048, 2048),
             (2049, 2049), (2050, 8191), (8192, 131_073), (8193, 131_073), (8193, 131_072), (6145, 3),
             (131_071, 5000), (131_072, 131_072), (131_073, 131_073), (140_001, 9000), (5, 131_073), (4096, 8192),
             (70, 1 << 22), (70, (1 << 22) + 1)]
    sets = [_elements(n, w, k) for k, (n, w) in enumerate(sizes) if n <= 60 * w]
    u = np.concatenate([np.full(len(s), k, np.uint32) for k, s in enumerate(sets)])
    v = np.concatenate(sets)
    t = eh.Trie(u, v, policy=2, forced=layout)
    probe = np.unique(np.concatenate([v[::7], v[::7] + 1]))
    for k, s in enumerate(sets):
        one = eh.Trie(np.zeros(len(s), np.uint32), s, policy=2, forced=UINT)
        one.relayout(policy=2, forced=layout)
        got, lay = t.set_bytes(k)
        want, _ = one.set_bytes(0)
        assert lay == layout
        np.testing.assert_array_equal(got, want)
        if layout == RANGE:  # number of words, first word, the words, their ranks
            words = np.zeros(int(s[-1] >> 6) - int(s[0] >> 6) + 1, np.uint64)
            np.bitwise_or.at(words, (s >> 6) - (s[0] >> 6), np.uint64(1) << (s & 63).astype(np.uint64))
            assert words.tobytes() in got.tobytes()
        one.free()
    # membership through the structures (their ranks place the rows of a pair's result)
    pairs = [(k, len(sets)) for k in range(len(sets))]
    counts, found = eh.set_intersect(sets + [probe], [layout] * len(sets) + [UINT], pairs, materialize=True)
    for s, c, f in zip(sets, counts, found):
        want = np.intersect1d(s, probe)
        assert c == len(want)
        np.testing.assert_array_equal(f, want)
    t.free()


def test_many_wide_thin_sets(eh):
    """256 sets of 50 elements over 9.6 M ids each: built one after the other, with
    three waits each, they would take over 10 ms."""
    sets = [_elements(50, 150_000, k) for k in range(256)]
    u = np.concatenate([np.full(50, k, np.uint32) for k in range(256)])
    t = eh.Trie(u, np.concatenate(sets), policy=2, forced=UINT)
    best = 1.0
    for _ in range(5):
        t.relayout(policy=2, forced=UINT)
        t0 = time.perf_counter()
        t.relayout(policy=2, forced=RANGE)
        best = min(best, time.perf_counter() - t0)
    assert best < 0.008, best
    t.free()
