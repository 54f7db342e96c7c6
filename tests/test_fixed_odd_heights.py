"""Owned chunks with a forced block of 512 threads on grids of up to 1024 groups
whose odd height makes more chunks than the block has warps, beside grids that
just fit: the walked schedule's bits, and larger grids refused."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(124, 33), (61, 61), (1364, 3), (4096, 1), (250, 15), (64, 63)])
def test_odd_heights_run_on_512_threads(W, H):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W + H, n_models=5, steps=30,
                                              W=W, H=H, n_exp=2)
    out = []
    for sched in (grn.SCHEDULE_WALK_ITEMS, grn.SCHEDULE_FIXED_ITEMS):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, threads=512)
            raw, states = ev.evaluate_states(batch, max_planes=8)
            st = ev.evaluate_batch(batch)[2]
        assert (st["schedule"], st["threads_per_block"]) == (sched, 512)
        out.append((raw, states, st["total_steps"]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


def test_more_than_two_groups_a_thread_are_refused():
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=1, n_models=2, steps=5, W=128,
                                              H=33)
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(grn.SCHEDULE_FIXED_ITEMS, threads=512)
        with pytest.raises(grn.GrnError) as e:
            ev.evaluate_batch(batch)
        assert e.value.status == 6  # GRN_ERR_CAPACITY
