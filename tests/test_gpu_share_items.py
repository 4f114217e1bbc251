"""The split of a triangle COUNT's work items over ranks: even also where most
items are shared by neighbouring entries (a sparse, even relation), and cut from
the relation and the schedule alone, so that ranks on which fewer warps are
resident (here: more staging per warp, without block items) still cut the same
items.  The shares run one after another on this GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _er(n, m, seed, sym):
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    u, v = u[u != v], v[u != v]
    if sym:
        return np.concatenate([u, v]), np.concatenate([v, u])
    return np.minimum(u, v), np.maximum(u, v)


@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("world", [2, 3, 4, 8, 16])
def test_shared_items_are_dealt_out(eh, world, sym):
    t = eh.Trie(*_er(1 << 17, 8 << 17, 1, sym))
    want, st = t.count("triangle", stats=True)
    # entries share items at all: unshared, every entry with rows has its own
    _, own = t.count("triangle", stats=True, record=True)
    assert st["work_items"] < 0.5 * own["work_items"]
    got = [t.count("triangle", shard=(r, world), stats=True) for r in range(world)]
    assert sum(c for c, _ in got) == want
    items = [s["work_items"] for _, s in got]
    assert max(items) < 1.1 * min(items), items
    t.free()


@pytest.mark.parametrize("n,m", [(12_000, 60_000), (40_000, 200_000)])
def test_ranks_of_unlike_devices_cut_the_same_items(eh, oracle, n, m):
    u, v = _er(n, m, 5, False)
    t = eh.Trie(u, v)
    want = oracle.Trie(u, v).triangle()
    assert want > 50
    kinds = (dict(), dict(smem_words=16384), dict(smem_words=64))
    got = [[t.count("triangle", shard=(r, 3), block_items=False, **k) for r in range(3)] for k in kinds]
    assert got[0] == got[1] == got[2]
    assert sum(got[0]) == want
    t.free()
