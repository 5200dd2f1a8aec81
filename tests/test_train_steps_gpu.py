"""Training of sixteen steps and more runs its weight gradients and column sums on
side streams, shorter training on one stream. With one step an epoch, every epoch's
loss is that of the parameters all steps before have made: sixteen steps beside
fifteen, the first fifteen losses are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,R,batch", [(8, 256, 1), (96, 1024, 1024), (104, 512, 130), (256, 2048, 33)])
def test_forked_steps_equal_single_stream_steps(d, R, batch):
    from parallel_anns_b200 import learned as LE
    rng = np.random.default_rng(d + R)
    X = rng.standard_normal((batch, d)).astype(np.float32)
    cells = rng.integers(0, R, (batch, 5)).astype(np.uint16)
    y = rng.uniform(4, 7, batch).astype(np.float32)
    one, few = LE.train(X, cells, y, R, epochs=15, batch=batch, seed=3)
    more, many = LE.train(X, cells, y, R, epochs=16, batch=batch, seed=3)
    assert np.array_equal(few, many[:15]) and np.unique(many).size == 16
    assert not np.array_equal(one, more)
