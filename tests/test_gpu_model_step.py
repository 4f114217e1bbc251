"""The one-kernel training step of small networks (and the per-layer kernels
above its size) against the double-precision oracle: batches that end inside a
block's rows, one sample, several passes of a block, one to four layers, a
network too wide for shared memory.  Tolerance: sums of the batch in fp32 pieces
of 16 rows and a 64-bit sum of those, over chains of at most 128 inputs:
|err| <= 2e-5 + 1e-4 |ref|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATOL, RTOL = 2e-5, 1e-4


@pytest.mark.parametrize("dims", [[6, 32, 32, 1], [3, 2], [5, 64, 7, 3], [4, 8, 8, 8, 2], [16, 128, 128, 1]])
@pytest.mark.parametrize("batch", [1, 15, 16, 17, 300, 5000])
def test_gradient_and_step(eh, oracle, dims, batch):
    rng = np.random.default_rng(batch)
    x = rng.normal(0, 1, (batch, dims[0])).astype(np.float32)
    y = rng.normal(0, 1, (batch, dims[-1])).astype(np.float32)
    m = eh.Model(dims, seed=3)
    p = m.params()
    want_loss, want = oracle.mlp_loss_grad(dims, p.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    loss, g = m.loss_grad(x, y)
    assert abs(loss - want_loss) <= ATOL + RTOL * abs(want_loss)
    np.testing.assert_allclose(g, want, rtol=RTOL, atol=ATOL)
    assert m.train(x, y, lr=0.05, steps=1) == pytest.approx(want_loss, rel=RTOL, abs=ATOL)
    np.testing.assert_allclose(m.params(), p - 0.05 * want, rtol=RTOL, atol=ATOL)
    a, b = eh.Model(dims, seed=3), eh.Model(dims, seed=3)
    la = a.train(x, y, lr=0.01, steps=3)
    for _ in range(3):
        lb = b.train(x, y, lr=0.01, steps=1)
    if dims[1] < 128:  # the small path sums in a fixed order
        assert la == lb
        np.testing.assert_array_equal(a.params(), b.params())
    for k in (m, a, b):
        k.free()
