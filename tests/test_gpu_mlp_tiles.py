"""The tensor-core trainer over one, two and several tiles per block: the
gradient of a batch is the mean of its tiles' own gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NIN = 24


@pytest.mark.parametrize("ntiles", [1, 128, 256, 512])
def test_batch_gradient_is_the_mean_of_its_tiles(ntiles):
    """Tiles of three kinds; a block's consecutive tiles (the SM count apart)
    differ unless that count is a multiple of three.  The batch sizes are
    powers of two, so 1/batch scales every BF16 operand exactly, and what is
    left is the FP32 accumulation: at most 32 MMA steps per block and 152
    partials of terms whose magnitudes add up to some 12 times the gradient,
    (32 * 2^-23 + 152 * 2^-24) * 12 = 1.6e-4 of the largest entry.  A tile
    left out, added twice or taken with another tile's inputs is off by a
    tenth or more."""
    from tmcore_gb300.gpu import ClosureMLP

    net = ClosureMLP(seed=7)
    net.set_train_mode(True)
    rng = np.random.default_rng(2)
    kx = rng.standard_normal((3, 128, NIN)).astype(np.float32)
    kt = (np.sin(kx[..., 0]) + 0.3 * kx[..., 5] + np.arange(3)[:, None]).astype(np.float32)
    one = [net.gradient(kx[k], kt[k]) for k in range(3)]
    kind = np.arange(ntiles) % 3
    g, loss = net.gradient(kx[kind].reshape(-1, NIN), kt[kind].reshape(-1))
    want = sum(one[k][0].astype(np.float64) * np.mean(kind == k) for k in range(3))
    mean = sum(one[k][1] * np.mean(kind == k) for k in range(3))
    assert np.max(np.abs(g - want)) <= 1.6e-4 * np.max(np.abs(want))
    assert abs(loss - mean) <= 1e-5 * mean
    net.close()
