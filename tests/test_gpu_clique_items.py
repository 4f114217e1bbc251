"""Work items of a 4-clique that runs without hit masks (selections, general
relations) stay as fine as they were before items grew with the work: the weight of a
row says little of its pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["sym", "general"])
def test_items_stay_fine(eh, kind):
    rng = np.random.default_rng(2)
    n, m = 70_000, 200_000  # a hub next to all: two thousand million candidates
    a, b = rng.integers(1, n, m), rng.integers(1, n, m)
    u = np.concatenate([np.zeros(n - 1, np.int64), np.minimum(a, b)[a != b]])
    v = np.concatenate([np.arange(1, n), np.maximum(a, b)[a != b]])
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    else:
        u, v = np.append(u, 5), np.append(v, 0)
    t = eh.Trie(u.astype(np.uint32), v.astype(np.uint32))
    if kind == "sym":
        got, st = t.count_select("clique4_sel", 7, stats=True)
        fine, fst = t.count_select("clique4_sel", 7, stats=True, config=dict(chunk=32768))
    else:
        got, st = t.count("clique4", stats=True)
        fine, fst = t.count("clique4", stats=True, chunk=32768)
    assert got == fine
    assert st["wedges"] > 1.9e9  # enough for larger items
    assert st["work_items"] >= fst["work_items"]
    t.free()
