"""The cost model's training kernels at the edges of their tiles: rows per CTA
(8), gradient slots (64), the size above which the slots are summed by a
kernel of their own (1024), and the smallest and largest feature counts.

Gradients against the FP64 oracle to 1e-4 of the largest, the bar of the
other cost-model tests: FP32 sums of up to 1100 terms, each layer's rounding
passed on to the next.  One Adam step against the formula on the device's own
gradient to 2e-7: the step is at most lr = 1e-3 with a few FP32 roundings, and
the weights are below 4 (one rounding: 2.4e-7 at most, half of that here)."""
import numpy as np
import pytest

from oracle import mlp
from qcs_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features,rows", [(20, 1), (20, 7), (20, 8), (20, 9), (1, 63), (7, 64),
                                           (20, 65), (64, 200), (20, 1024), (20, 1025),
                                           (8, 1100)])
def test_gradients_and_one_adam_step(features, rows):
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, features)).astype(np.float32)
    y = rng.normal(size=rows).astype(np.float32)
    m = capi.CostModel(seed=rows, features=features)
    p = m.params()
    loss, g = m.loss_grad(x, y)
    ref_loss, ref_g = mlp.loss_grad(p.astype(np.float64), x, y, features)
    assert abs(loss - ref_loss) <= 1e-5 * max(1.0, ref_loss)
    assert np.max(np.abs(g - ref_g)) <= 1e-4 * np.max(np.abs(ref_g))
    np.testing.assert_allclose(m.predict(x), mlp.forward(p, x, features), rtol=1e-4, atol=1e-4)
    m.train(x, y, epochs=1, batch=rows, lr=1e-3)
    b1, b2, lr = (float(np.float32(v)) for v in (0.9, 0.999, 1e-3))
    gd = g.astype(np.float64)
    mm, vv = (1 - b1) * gd, (1 - b2) * gd * gd
    want = p - lr * (mm / (1 - b1)) / (np.sqrt(vv / (1 - b2)) + 1e-8)
    assert np.max(np.abs(m.params() - want)) <= 2e-7
    m.close()
