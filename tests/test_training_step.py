"""The training step's launches at the sizes where they can go wrong: batches
around a tile and a K slice, weight gradients in one K range and in several
(which the Adam kernel adds itself).  Adam's first step from zero moments
moves a weight by lr * g / (|g| + 1e-8), so each weight whose gradient is not
lost in rounding must move by lr against the sign that the gradient call, which
adds its K ranges in a kernel of its own, gives for the same rows."""
import numpy as np
import pytest

import grn_b200 as grn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 128, 255, 257, 513, 8192])
def test_first_step_follows_the_gradient(rows):
    rng = np.random.default_rng(rows)
    x = rng.uniform(0, 1, (rows, grn.N_FEATURES)).astype(np.float32)
    t = rng.normal(-1, 0.5, rows).astype(np.float32)
    lr = 1e-3
    for tcgen05 in (True, False):
        sur = grn.Surrogate(seed=3, capacity=max(rows, 64))
        sur.use_tcgen05(tcgen05)
        w0 = sur.params()
        loss, g = sur.gradients(x, t)
        sur.add_data(x, t)
        mean = sur.train(epochs=1, batch_size=rows, lr=lr)
        moved = sur.params() - w0
        assert abs(mean - loss) <= 1e-6 * abs(loss) + 1e-12  # the rows in another order
        # FP32 sums of `rows` BF16 products in another order differ by less
        # than rows * 2^-24 of the sum of magnitudes; 2e-2 of the largest
        # gradient is far above that and above the 1e-8 in Adam's divisor.
        clear = np.abs(g) > 2e-2 * np.abs(g).max()
        assert clear.sum() > 50
        # Each weight is rounded once to FP32 after the step (|w| < 1: 2^-24).
        assert np.abs(moved[clear] + lr * np.sign(g[clear])).max() <= 1e-2 * lr
        assert np.abs(moved[g == 0]).max(initial=0.0) == 0.0
        sur.close()
