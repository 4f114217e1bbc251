"""eh_query_stats.launches counts every kernel of a query: of the plans on hit
masks the mask plan's, and the launches that only some relations need (4-cliques of
parts past 32 and past 2048 elements, annotation of parts past 4096)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLAN = 3  # kernels that make the items


def _hub(d, kind):
    """Vertex 0 next to 1..d, a path through those: triangles, no 4-clique."""
    u = np.concatenate([np.zeros(d, np.int64), np.arange(1, d)]).astype(np.uint32)
    v = np.concatenate([np.arange(1, d + 1), np.arange(2, d + 1)]).astype(np.uint32)
    return (u, v) if kind == "up" else (np.concatenate([u, v]), np.concatenate([v, u]))


def _scans(n):
    """Kernels of a scan of n values: one tile of 2048, or tile sums, their scan, and the tiles."""
    tiles = -(-n // 2048)
    return 1 if tiles == 1 else 2 + _scans(tiles)


@pytest.mark.parametrize("d,passes", [(40, 3), (2048, 3), (2080, 4), (4096, 4), (4200, 4)])
def test_clique_launches(eh, d, passes):
    t = eh.Trie(*_hub(d, "up"))
    heads = t.info()["n_head"]
    c, st = t.count("clique4", stats=True)
    assert c == 0
    assert st["launches"] == 1 + _scans(heads) + _scans(heads + 1) + PLAN + passes
    b = eh.Batch([t, t], "clique4")
    assert b.run(stats=True)[1]["launches"] == passes
    b.free()
    b = eh.Batch([t, t], "triangle")
    assert b.run(stats=True)[1]["launches"] == 1
    b.free()
    t.free()


@pytest.mark.parametrize("d,passes", [(40, 2), (4096, 2), (4200, 3)])
def test_annotation_launches(eh, d, passes):
    t = eh.Trie(*_hub(d, "sym"))
    heads = t.info()["n_head"]
    c, st = t.count("lollipop", stats=True)
    assert c == 2 * (d - 1) * d + 2 * (2 * 1 * 2 + (d - 2) * 2 * 3)  # hub, path ends, path
    # the root bag is one more
    assert st["launches"] == 1 + _scans(heads) + _scans(heads + 1) + PLAN + passes + 1
    t.free()
