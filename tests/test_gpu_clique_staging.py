"""A 4-clique asked for with more staging than a block may have is refused, on every
relation and whichever plan it runs, as it is by the entry that allocates nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["up", "down", "sym", "general", "no_candidates"])
def test_refused(eh, kind):
    u, v = (np.asarray(x, np.uint32) for x in np.triu_indices(30, 1))
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    if kind == "general":
        u, v = np.concatenate([u, v[:7]]), np.concatenate([v, u[:7]])
    if kind == "no_candidates":
        u, v = u[:1], v[:1]
    t = eh.Trie(u, v)
    want = t.count("clique4")
    for kw in (dict(smem_words=1 << 20), dict(smem_words=8192, warps=16)):
        with pytest.raises(eh.EHError, match="staging exceeds"):
            t.count("clique4", **kw)
        with pytest.raises(eh.EHError, match="staging exceeds"):
            eh.Batch([t, t], "clique4", config=kw)
        assert t.count("triangle", **kw) == t.count("triangle")  # shrinks instead
    assert t.count("clique4", smem_words=8192, warps=4) == want
    assert t.count("clique4") == want
    t.free()
