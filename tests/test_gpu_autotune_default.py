"""The autotuner starts from the schedule that a query without one runs."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [10, 14, 18])
def test_default_is_the_engines(eh, scale):
    from emptyheaded_b200 import autotune
    u, v = eh.gen_rmat(3, scale, 16 << scale)
    s, d, _ = eh.preprocess(u, v)
    t = eh.Trie(s, d)
    want, st = t.count("triangle", stats=True)
    got, cst = t.count("triangle", stats=True, config=autotune.DEFAULT)
    assert got == want
    assert cst["work_items"] == st["work_items"]
    assert autotune.DEFAULT["chunk"] in autotune.GRID["chunk"]
    t.free()
