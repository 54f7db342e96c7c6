"""Models that come to rest (every rate exactly 0) on steps without a block
barrier stop within a few dozen steps of it instead of running to the last one,
with the step count of the first step without a rate, on one CTA and on a
cluster; a negative threshold runs every step."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu

STEPS = 4_000_000


def _rest(W, H, sched, cluster, steps, threshold=0.0):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=3, n_models=4, steps=steps,
                                              W=W, H=H, n_exp=2)
    params["min_conc_change"] = threshold
    for k in ("lim", "dif"):
        batch.products[k] = 0.0
    batch.products["deg"] = 1.0  # half of what is left goes in a step
    params["dt"] = 0.5
    init[1] = 0.0                # at rest from the first step
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(sched, cluster_size=cluster)
        _, raw, st = ev.evaluate_batch(batch)
        assert st["schedule"] == sched
    return raw, st


@pytest.mark.parametrize("W,H,sched,cluster", [
    (64, 64, grn.SCHEDULE_FIXED_ITEMS, 0), (8, 8, grn.SCHEDULE_FIXED_ITEMS, 0),
    (64, 64, grn.SCHEDULE_CLUSTER, 4),
])
def test_a_model_at_rest_stops(W, H, sched, cluster):
    raw, st = _rest(W, H, sched, cluster, STEPS)
    # A step takes at least 0.3 us: to the last one that would be 1.2 s an
    # experiment.  Halving 1.0 down to 0 takes about 150 steps.
    assert st["kernel_ms"] < 100
    walk_raw, walk = _rest(W, H, grn.SCHEDULE_WALK_ITEMS, 0, STEPS)
    assert st["total_steps"] == walk["total_steps"]
    assert np.array_equal(raw, walk_raw)


@pytest.mark.parametrize("steps", [1, 2, 63, 64, 65, 128, 129, 200])
def test_step_counts_around_a_vote(steps):
    for threshold in (0.0, -1.0):
        out = [_rest(16, 16, s, c, steps, threshold)
               for s, c in ((grn.SCHEDULE_FIXED_ITEMS, 0), (grn.SCHEDULE_WALK_ITEMS, 0),
                            (grn.SCHEDULE_CLUSTER, 2))]
        for raw, st in out[1:]:
            assert st["total_steps"] == out[0][1]["total_steps"]
            assert np.array_equal(raw, out[0][0])
        if threshold < 0:
            assert out[0][1]["total_steps"] == 4 * 2 * steps
