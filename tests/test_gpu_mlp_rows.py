"""Cost-model gradients over more rows than are kept at a time (2^18): at that edge,
and above 65535 slots of 64 rows.

Up to 5.3e5 rows: against the FP64 oracle, to 1e-4 of the largest as in
test_gpu_mlp.py.  The largest repeats 128 rows, so that the oracle of those is the
whole's; its 65538 slots, of two kinds, are summed one after another in FP32, which
rounds by at most 2^-24 of the sum of their magnitudes each time."""
import numpy as np
import pytest

from oracle import mlp
from qcs_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [262143, 262144, 262145, 262144 + 64, 524288 + 70])
def test_rows_in_pieces(rows):
    r = np.random.default_rng(rows)
    x = r.normal(size=(rows, 3)).astype(np.float32)
    y = r.normal(size=rows).astype(np.float32)
    m = capi.CostModel(seed=4, features=3)
    loss, g = m.loss_grad(x, y)
    ref_loss, ref_g = mlp.loss_grad(m.params().astype(np.float64), x, y, 3)
    assert abs(loss - ref_loss) <= 1e-5 * max(1.0, ref_loss)
    assert np.max(np.abs(g - ref_g)) <= 1e-4 * np.max(np.abs(ref_g))
    # one step on all rows is Adam's on this gradient (its first step: lr * sign)
    p = m.params()
    m.train(x, y, epochs=1, batch=rows, lr=1e-3)
    gd = g.astype(np.float64)
    lr, b1, b2 = (float(np.float32(v)) for v in (1e-3, 0.9, 0.999))
    want = p - lr * ((1 - b1) * gd / (1 - b1)) / (np.sqrt((1 - b2) * gd * gd / (1 - b2)) + 1e-8)
    assert np.max(np.abs(m.params() - want)) <= 2e-7
    m.close()


def test_more_slots_than_a_grid_dimension():
    repeat, half = 32769, 64
    r = np.random.default_rng(5)
    x = r.normal(size=(2 * half, 2)).astype(np.float32)
    y = r.normal(size=2 * half).astype(np.float32)
    m = capi.CostModel(seed=2, features=2)
    p = m.params().astype(np.float64)
    loss, g = m.loss_grad(np.tile(x, (repeat, 1)), np.tile(y, repeat))
    ref_loss, ref_g = mlp.loss_grad(p, x, y, 2)
    parts = [np.abs(mlp.loss_grad(p, x[k:k + half], y[k:k + half], 2)[1]) for k in (0, half)]
    assert abs(loss - ref_loss) <= 1e-5 * max(1.0, ref_loss)
    bound = 1e-4 * np.max(np.abs(ref_g)) + (2 * repeat) * 2.0 ** -24 * (parts[0] + parts[1]) / 2
    assert np.all(np.abs(g - ref_g) <= bound)
    m.close()
