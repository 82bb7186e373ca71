"""The network's activation far out on its tails: z sigmoid(z) of a large
negative z is 0 (as z / (1 + exp(-z)) in FP32, whose exponential overflows), not
a number that later weights can make visible; a pre-activation that has
overflowed gives NaN."""
import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def chain(w1, w2):
    """Parameters of one path through the network: f0 -> w1 -> w2 -> 1 -> 1, all others 0."""
    th = np.zeros(mo.NPARAMS, np.float32)
    th[[mo.OFF_W1, mo.OFF_W2, mo.OFF_W3, mo.OFF_W4]] = w1, w2, 1.0, 1.0
    return th


def predict(w1, w2, f0=1.0):
    from channel_gb300.closure import Mlp

    with Mlp(0) as m:
        m.norm = {"mu_in": np.zeros(10), "sd_in": np.ones(10), "mu_out": np.zeros(6), "sd_out": np.ones(6)}
        m.params = chain(w1, w2)
        feat = np.zeros((10, 256), np.float32)
        feat[0] = f0
        return m.predict(feat)[0]


@pytest.mark.parametrize("z", [-89.0, -100.0, -1000.0, -3e38])
def test_saturated_activation_is_zero(gpu_lib, z):
    assert np.all(predict(z, 1e36) == 0.0)


@pytest.mark.parametrize("z", [-60.0, -80.0, -87.0])
def test_small_activations(gpu_lib, z):
    """Down to the smallest normal number; BF16 operands, three roundings of 2^-9."""
    h = z / (1.0 + np.exp(-z))
    w2 = -1.0 / h
    h2 = -1.0 / (1.0 + np.e)
    h3 = h2 / (1.0 + np.exp(-h2))
    np.testing.assert_allclose(predict(z, w2), h3, rtol=4 * 2.0**-9)


def test_overflowed_pre_activation_is_nan(gpu_lib):
    assert np.isnan(predict(-3e38, 1.0, f0=100.0)).all()
