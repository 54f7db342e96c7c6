"""State planes padded after every row of strips (rows of groups that a warp's
accesses cross) against planes without padding (all in global memory): owned
and walked chunks, and clusters whose bands have odd heights, so that an edge
row moves by a different number of bytes up and down.  The same bits, with and
without a step barrier (early-exit threshold)."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,cluster", [
    (20, 22, 2), (51, 37, 2), (36, 26, 4), (12, 40, 8), (5, 31, 2), (100, 11, 4),
])
@pytest.mark.parametrize("threshold", [0.0, 1e-3])
def test_padded_planes_give_the_same_states(W, H, cluster, threshold):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W * 7 + H, n_models=12,
                                              steps=60, W=W, H=H, genes=(2, 7), links=(2, 20),
                                              n_exp=2)
    params["min_conc_change"] = threshold
    out = []
    for sched, c in ((grn.SCHEDULE_GLOBAL, 0), (grn.SCHEDULE_FIXED_ITEMS, 0),
                     (grn.SCHEDULE_WALK_ITEMS, 0), (grn.SCHEDULE_CLUSTER, cluster)):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, cluster_size=c)
            raw, states = ev.evaluate_states(batch, max_planes=16)
            _, _, st = ev.evaluate_batch(batch)
        assert st["schedule"] == sched
        out.append((raw, states, st["total_steps"]))
    for raw, states, total in out[1:]:
        assert np.array_equal(states, out[0][1]) and np.array_equal(raw, out[0][0])
        assert total == out[0][2]
