"""Training calls of few steps run their captured step on one stream, longer ones on three: the same
kernels and sums, so a training cut into short calls is the one long call, bit for bit."""
import numpy as np
import pytest

from mind_b200 import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,hidden,batch", [(1, 16, 33), (2, 256, 700), (6, 64, 2500)])
def test_short_calls_equal_one_long_call(layers, hidden, batch):
    rng = np.random.default_rng(layers)
    x = rng.normal(0.0, 1.0, (900, 70)).astype(np.float32)
    y = (rng.uniform(size=900) < 0.3).astype(np.float32)
    runs = []
    for calls in ([70], [31, 32, 7], [1] * 4 + [30, 36]):
        net = surrogate.Mlp(n_in=70, hidden=hidden, layers=layers, seed=8)
        losses = np.concatenate([net.train(x, y, steps=n, batch=batch)[0] for n in calls])
        runs.append((losses, net.params))
        net.close()
    for losses, params in runs[1:]:
        assert np.array_equal(losses, runs[0][0]) and np.array_equal(params, runs[0][1])


def test_no_training_without_a_training_set():
    """A set too large for the device is refused, and takes the one before it along: a training call
    after it is refused as well, until there is a set again."""
    rng = np.random.default_rng(0)
    x = rng.normal(0.0, 1.0, (64, 70)).astype(np.float32)
    y = (rng.uniform(size=64) < 0.3).astype(np.float32)
    net = surrogate.Mlp(n_in=70, hidden=16, layers=1, seed=8)
    net.train(x, y, steps=2, batch=32)
    lib, f32 = net.lib, surrogate._f32
    assert lib.mind_mlp_set_data(net.handle, f32(x), f32(y), 1 << 40) == surrogate.abi.MIND_ECUDA
    assert lib.mind_mlp_train(net.handle, 2, 32, 1e-3, None, None) == surrogate.abi.MIND_EARG
    losses, _ = net.train(x, y, steps=2, batch=32)
    assert np.all(np.isfinite(losses))
    net.close()
