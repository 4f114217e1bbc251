"""Plans on hit masks where the head entries that have work units lie far apart:
two dense groups of vertices with a long path of ids between them, whose entries
have none.  The warps that go from one group to the other look the next entry up
instead of walking: 400,000 loads, one after the other, would take over 10 ms
(25 ns each at the very least), the whole query takes well under one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, PATH = 40, 400_000


def _relation(sym):
    u, v = np.triu_indices(D, 1)
    p = np.arange(100, 100 + PATH)
    far = 1_000_000
    u, v = np.concatenate([u, p, u + far]), np.concatenate([v, p + 1, v + far])
    if sym:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u.astype(np.uint32), v.astype(np.uint32)


@pytest.mark.parametrize("sym", [False, True])
def test_units_far_apart(eh, sym):
    t = eh.Trie(*_relation(sym))
    cliques = 2 * (D * (D - 1) * (D - 2) * (D - 3) // 24) * (24 if sym else 1)
    got = [t.count("clique4", stats=True) for _ in range(5)]
    assert [c for c, _ in got] == [cliques] * 5
    assert min(st["kernel_ms"] for _, st in got) < 4.0
    b = eh.Batch([t, t], "clique4")
    got = [b.run(stats=True) for _ in range(5)]
    assert all(c.tolist() == [cliques] * 2 for c, _ in got)
    assert min(st["kernel_ms"] for _, st in got) < 4.0
    b.free()
    if sym:
        # sum over a of T(a) d(a); T = (d - 1) (d - 2) in a group of D, 0 on the path
        got = [t.count("lollipop", stats=True) for _ in range(5)]
        assert [c for c, _ in got] == [2 * D * (D - 1) * (D - 2) * (D - 1)] * 5
        assert min(st["kernel_ms"] for _, st in got) < 4.0
    t.free()
