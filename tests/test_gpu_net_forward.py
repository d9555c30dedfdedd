"""The forecaster's forward pass on more samples than its launch has CTAs (two
per SM, 296), each of which then takes several: a sample's logit is the same bits
in any batch, so it equals that of the same samples in small batches."""
import numpy as np
import pytest

import amrlbm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [297, 1000])
def test_large_batches(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 4, 18, 18)).astype(np.float32)
    with amrlbm.Net(seed=4, max_batch=n) as net:
        z = net.forward(x)
    with amrlbm.Net(seed=4, max_batch=64) as net:
        small = np.concatenate([net.forward(x[i:i + 64]) for i in range(0, n, 64)])
    assert len(np.unique(z)) > n // 2  # not one value for all
    assert np.array_equal(z, small)
