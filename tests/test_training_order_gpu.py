"""The order in which training takes its rows, against a shuffle on the CPU."""
import numpy as np
import pytest

from oracle import mlp_ref
from pbf_gb300 import mlp_fit_normalization, mlp_init, mlp_params, mlp_train

pytestmark = pytest.mark.gpu


def shuffled_rows(rows, seed):
    """The training's row order: a Fisher-Yates shuffle, from the last entry
    down, with the draws of a splitmix64 stream."""
    mask = (1 << 64) - 1
    s, order = seed ^ 0x5EED, list(range(rows))
    for i in range(rows - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return np.array(order)


@pytest.mark.parametrize("rows,batch", [(1, 1), (2, 1), (257, 64), (4099, 1000)])
def test_training_takes_the_rows_in_shuffled_order(rows, batch):
    """With a step of 0 the network stays, and the loss handed back is the mean
    over the last whole batch: it names the rows of that batch.  1e-3 is the
    bound of the loss against FP64 with the same bf16 rounding points."""
    rng = np.random.default_rng(21)
    feat = rng.normal(size=(rows, 8)).astype(np.float32)
    target = (feat[:, 0] * np.exp(rng.normal(size=rows))).astype(np.float32)
    m = mlp_init(21)
    mlp_fit_normalization(m, feat, target)
    mean, istd, scale = (np.ctypeslib.as_array(m.feat_mean).copy(), np.ctypeslib.as_array(m.feat_inv_std).copy(),
                         float(m.lam_scale))
    before = mlp_params(m).copy()
    loss = mlp_train(m, feat, target, epochs=1, batch=batch, lr=0.0, seed=2 ** 63 + rows)
    assert np.array_equal(mlp_params(m), before)
    last = rows // batch * batch
    pick = shuffled_rows(rows, 2 ** 63 + rows)[last - batch:last]
    _, want = mlp_ref.gradient(before, mean, istd, scale, feat[pick], target[pick], emulate=True)
    assert abs(loss - want) <= 1e-3 * max(want, 1e-12)
