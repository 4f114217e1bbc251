"""The trie build over rows that arrive in order (not sorted again), in order
with repeats, and out of order, at lengths around the tiles of the CSR pass, the
scan and the sort, for relations of every direction: contents and counts against
the oracle; integer work, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, kind, seed):
    rng = np.random.default_rng(seed)
    span = max(4, int(n ** 0.6))
    u = rng.integers(0, span, 2 * n).astype(np.uint32)
    v = (rng.integers(0, 3 * span, 2 * n)).astype(np.uint32)
    if kind != "general":
        keep = u != v
        u, v = np.minimum(u, v)[keep], np.maximum(u, v)[keep]
        if kind == "down":
            u, v = v, u
        elif kind == "sym":
            u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u[:n] if kind != "sym" else u, v[:n] if kind != "sym" else v


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general"])
@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 4095, 4096, 4097, 30000])
def test_orders_of_arrival(eh, oracle, kind, n):
    u, v = _rows(n, kind, n)
    if not len(u):
        return
    o = oracle.Trie(u, v)
    order = np.lexsort((v, u))
    rep = np.repeat(order, 1 + (np.arange(len(order)) % 3 == 0))
    last = order.copy()
    last[-2:] = last[-2:][::-1]  # only the last two rows out of order
    for idx in (np.arange(len(u)), order, rep, np.unique(np.stack([u, v], 1), axis=0, return_index=True)[1], last,
                order[::-1]):
        t = eh.Trie(u[idx], v[idx])
        head, off, vals, _ = t.export()
        np.testing.assert_array_equal(head, o.head)
        np.testing.assert_array_equal(off, o.off)
        np.testing.assert_array_equal(vals, o.vals)
        assert t.info()["n_nodes"] == max(u.max(), v.max()) + 1
        assert t.count("triangle") == o.triangle()
        t.free()


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 4097, 100000])
def test_preprocess_and_encode_lengths(eh, oracle, n):
    u, v = eh.gen_rmat(3, 12, n)
    s, d, nodes = eh.preprocess(u, v)
    ou, ov = oracle.gen_rmat(3, 12, n)
    os_, od, on = oracle.preprocess(ou, ov)
    np.testing.assert_array_equal(s.numpy(), os_)
    np.testing.assert_array_equal(d.numpy(), od)
    assert nodes == on
    x = np.random.default_rng(n).integers(-(1 << 50), 1 << 50, n)
    x = np.concatenate([x, x[: n // 2]])
    enc = eh.Encoding([x], "int64")
    want, keys = np.unique(x, return_inverse=True)
    np.testing.assert_array_equal(enc.values(), want)
    np.testing.assert_array_equal(enc.encode(x), keys)
    enc.free()
