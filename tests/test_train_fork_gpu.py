"""Training runs of sixteen steps and more (R up to 2,048) compute weight gradients and column
sums on side streams; shorter runs use one stream. Both give the same numbers: the
first epoch of a long run equals the same epoch as a run of its own, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,R,batch,steps", [(8, 256, 1, 15), (96, 1024, 1024, 10), (104, 512, 130, 15),
                                             (256, 2048, 33, 9), (16, 4096, 40, 9)])
def test_first_epoch_equals_short_run(d, R, batch, steps):
    from parallel_anns_b200 import learned as LE
    rng = np.random.default_rng(d + R)
    n = batch * steps
    X = rng.standard_normal((n, d)).astype(np.float32)
    cells = rng.integers(0, R, (n, 5)).astype(np.uint16)
    y = rng.uniform(4, 7, n).astype(np.float32)
    p1, short = LE.train(X, cells, y, R, epochs=1, batch=batch, seed=3)
    p2, long = LE.train(X, cells, y, R, epochs=2, batch=batch, seed=3)
    p3, again = LE.train(X, cells, y, R, epochs=2, batch=batch, seed=3)
    assert short[0] == long[0] and np.array_equal(long, again)
    assert np.array_equal(p2, p3) and not np.array_equal(p1, p2)
