"""Loss and gradient of the refine-flag forecaster on batches whose
324 n rows end inside a 16-row product step, inside a stage of the weight
gradient's rows or past several, with fewer and more samples than CTAs,
against the NumPy restatement with the same BF16 roundings. Tolerance: the
sums are FP32 over up to 324 n terms and the tensor core truncates as it
accumulates, at most 2^-23 per step of 16 rows, so 324 n / 16 * 1.2e-7 of the
sum of magnitudes (4e-4 at n = 150); 1e-3 of a parameter block's norm, as the
other gradient test allows."""
import numpy as np
import pytest

import amrlbm
import net_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 17, 150])
def test_batch_sizes(n):
    rng = np.random.default_rng(100 + n)
    x = rng.standard_normal((n, 4, 18, 18)).astype(np.float32)
    y = (rng.random(n) < 0.4).astype(np.float32)
    with amrlbm.Net(seed=3, max_batch=n) as net:
        p = net.params()
        loss, g = net.gradient(x, y, pos_weight=2.0)
        rl, rg, _ = net_ref.loss_and_grad(p, x, y, pos_weight=2.0)
        assert abs(loss - rl) <= 1e-4 * max(1.0, abs(rl))
        ends = (net_ref.O_W1, net_ref.O_B1, net_ref.O_W2, net_ref.O_B2, net_ref.O_W3, net_ref.O_B3,
                net_ref.O_WD, net_ref.O_BD, net_ref.NPARAM)
        for a, b in zip(ends, ends[1:]):
            err = np.linalg.norm(g[a:b] - rg[a:b]) / max(np.linalg.norm(rg[a:b]), 1e-12)
            assert err < 1e-3, (a, err)
