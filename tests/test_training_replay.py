"""Training steps replayed as a graph (the gather's first row, the Adam step and
the branches' joins all live on the device): each replay takes the rows that
follow, across epochs and chunks of indices, and gives the bits of a step
launched directly."""
import numpy as np
import pytest

import grn_b200 as grn

pytestmark = pytest.mark.gpu


def _data(rows, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (rows, grn.N_FEATURES)).astype(np.float32)
    # A few rows carry nearly all of the loss: rows left out or taken twice show.
    t = (rng.normal(size=rows) * 10.0 ** rng.uniform(-1, 3, rows)).astype(np.float32)
    return x, t


@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("rows,batch,epochs", [
    (5120, 512, 2), (640, 64, 3), (96, 96, 5),
    (8192, 512, 17),  # indices in two chunks (131072 at a time)
])
def test_each_replay_takes_its_own_rows(rows, batch, epochs, tcgen05):
    x, t = _data(rows, rows + batch)
    s = grn.Surrogate(seed=1, capacity=rows)
    s.use_tcgen05(tcgen05)
    s.add_data(x, t)
    # A learning rate that moves no weight: the mean over whole epochs of equal
    # minibatches is the mean over the rows.  Outputs are the same FP32 sums as
    # predictions, errors their FP32 differences, squares and sums FP64.
    want = np.mean((s.predict(x) - t).astype(np.float64) ** 2)
    mean = s.train(epochs=epochs, batch_size=batch, lr=1e-30)
    assert abs(mean - want) <= 1e-9 * want
    s.close()


@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("batch", [33, 512, 2048])
def test_replays_give_the_bits_of_direct_steps(batch, tcgen05):
    steps, lr = 6, 1e-3
    x, t = _data(3000, batch)
    replayed = grn.Surrogate(seed=5, capacity=3000)
    replayed.use_tcgen05(tcgen05)
    replayed.add_data(x, t)
    state = replayed.checkpoint()
    mean = replayed.train_batches(steps, batch, lr)
    # Every step by a surrogate of its own, whose first step is launched
    # directly.
    losses = []
    for _ in range(steps):
        one = grn.Surrogate(seed=9, capacity=3000)
        one.use_tcgen05(tcgen05)
        one.restore(state)
        losses.append(one.train_batches(1, batch, lr))
        state = one.checkpoint()
        direct = one.params()
        one.close()
    assert np.array_equal(replayed.params(), direct)
    assert replayed.checkpoint() == state  # moments, step and sampling too
    assert abs(mean - np.mean(losses)) <= 1e-12 * mean
    replayed.close()


def test_uneven_last_batches_and_epochs_in_one_call():
    """700 rows in batches of 256 (the last of 188), two epochs in one call or
    in two, and again: the same bits."""
    x, t = _data(700, 3)
    out = []
    for calls in ((2,), (1, 1), (2,)):
        s = grn.Surrogate(seed=6, capacity=700)
        s.add_data(x, t)
        for e in calls:
            s.train(epochs=e, batch_size=256, lr=1e-3)
        out.append(s.checkpoint())
        s.close()
    assert out[0] == out[1] == out[2]
