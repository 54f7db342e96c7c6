"""Forced block sizes of the streaming schedules: every whole number of warps up
to their own default runs, with the same bits; larger ones are refused."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sched", [grn.SCHEDULE_STREAM, grn.SCHEDULE_STREAM2])
def test_block_sizes_of_streaming(sched):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=8, n_models=5, steps=21, W=130,
                                              H=57, genes=(2, 9), links=(2, 20), n_exp=2)
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(sched)
        want, want_states = ev.evaluate_states(batch, max_planes=16)
        default = ev.evaluate_batch(batch)[2]["threads_per_block"]
        for threads in (32, 64, 224, 512, 608, default):
            ev.set_schedule(sched, threads=threads)
            raw, states = ev.evaluate_states(batch, max_planes=16)
            st = ev.evaluate_batch(batch)[2]
            assert (st["schedule"], st["threads_per_block"]) == (sched, threads)
            assert np.array_equal(raw, want) and np.array_equal(states, want_states)
        ev.set_schedule(sched, threads=default + 32)
        with pytest.raises(grn.GrnError) as e:
            ev.evaluate_batch(batch)
        assert e.value.status == 6  # GRN_ERR_CAPACITY
