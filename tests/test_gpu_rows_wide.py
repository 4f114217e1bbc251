"""Materialized triangles of wide, nearly empty neighbourhoods: a vertex next to
all others, a few edges among those, so its rows' masks are long and mostly zero.
The rows equal the oracle's, and getting them costs a small multiple of counting
them (the same intersections twice, counts and copies), not one wait per word."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(n, extra, kind):
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, extra), rng.integers(0, n, extra)
    u, v = np.concatenate([np.zeros(n - 1, np.int64), a]), np.concatenate([np.arange(1, n), b])
    keep = u != v
    u, v = np.minimum(u, v)[keep].astype(np.uint32), np.maximum(u, v)[keep].astype(np.uint32)
    return (u, v) if kind == "up" else (v, u)


@pytest.mark.parametrize("kind", ["up", "down"])
@pytest.mark.parametrize("n,extra", [(1020, 300), (1030, 9000), (3000, 200), (5000, 40000)])
def test_rows_of_wide_neighbourhoods(eh, oracle, kind, n, extra):
    u, v = _star(n, extra, kind)
    t = eh.Trie(u, v)
    np.testing.assert_array_equal(t.materialize(), oracle.Trie(u, v).triangle_tuples())
    t.free()


def test_time_of_wide_neighbourhoods(eh):
    t = eh.Trie(*_star(1 << 16, 1 << 18, "up"))

    def best(f):
        f()
        ts = []
        for _ in range(5):
            t0 = time.perf_counter()
            f()
            ts.append(time.perf_counter() - t0)
        return min(ts)

    assert best(t.materialize) < 6 * best(lambda: t.count("triangle"))
    t.free()
