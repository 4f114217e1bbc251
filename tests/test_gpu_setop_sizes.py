"""Set structures and intersections at the sizes where the work moves from a
warp to a block and to the grid: sets of 2047 to 2049 elements and words and of
131071 to 131073, pairs that stream 511 to 513 elements or words and several
rounds of a block, in every pair of layouts; exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BITSET, UINT, BLOCK = 0, 1, 3


@pytest.mark.parametrize("n", [511, 512, 513, 1023, 1025, 5000, 9000])
@pytest.mark.parametrize("la", [UINT, BITSET, BLOCK])
@pytest.mark.parametrize("lb", [UINT, BITSET, BLOCK])
def test_pair_sizes(eh, n, la, lb):
    rng = np.random.default_rng(n)
    sets = [np.sort(rng.choice(span, k, replace=False)).astype(np.uint32) + o
            for span, k, o in ((4 * n, n, 0), (4 * n, n, 7), (64 * n, n, 0), (64 * n, 3 * n, 65), (2 * n, 3, 0))]
    sets += [np.arange(n, dtype=np.uint32) * 64 + 5, np.zeros(0, np.uint32)]  # n words; empty
    k = len(sets)
    pairs = [(i, k + j) for i in range(k) for j in range(k)]
    counts, elems = eh.set_intersect(sets + sets, [la] * k + [lb] * k, pairs, materialize=True)
    for (i, j), c, e in zip(pairs, counts, elems):
        want = np.intersect1d(sets[i], sets[j - k])
        assert c == len(want), (i, j)
        np.testing.assert_array_equal(e, want)
    np.testing.assert_array_equal(eh.set_intersect(sets + sets, [la] * k + [lb] * k, pairs), counts)


@pytest.mark.parametrize("n", [2047, 2048, 2049, 131071, 131072, 131073])
@pytest.mark.parametrize("step", [1, 3, 64, 300])
def test_structure_bytes(eh, oracle, n, step):
    """Child sets of n elements, packed or a word or a block apart."""
    v = (np.arange(n, dtype=np.uint32) * step) + 11
    u = np.zeros(n, np.uint32)
    for forced in (BITSET, BLOCK):
        t = eh.Trie(u, v, policy=2, forced=forced, max_bitset_bytes=1 << 40)
        raw, lay = t.set_bytes(0)
        if lay == BITSET:
            want = np.array(oracle.range_bitset(v), np.uint8)
            w = (len(want) - 8) // 12
            words = want[8:8 + 8 * w].view(np.uint64)
            for r in (raw, want):  # ranks of empty words are unspecified in the reference's builder
                r[8 + 8 * w:].view(np.uint32)[words == 0] = 0
            np.testing.assert_array_equal(raw, want)
        else:
            np.testing.assert_array_equal(raw, oracle.block_bitset(v))
        t.free()
