"""Steps without a block barrier (owned chunks, fast models, no early-exit
threshold) against the walked and the cluster schedules, which pass a barrier
every step: the same states, errors and step counts.  Long thin and short
wide grids (a chunk's neighbours one and several chunks away), one step, and
models that stop because every rate is exactly 0 (all concentrations and
rates 0: after the first step) beside ones that run to the end."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,steps,genes", [
    (4, 250, 300, (2, 4)), (64, 64, 1, (2, 8)), (64, 64, 2, (2, 8)), (63, 30, 333, (3, 8)),
    (320, 6, 200, (2, 6)), (20, 20, 500, (2, 3)), (48, 48, 120, (9, 16)),
])
def test_matches_schedules_with_a_barrier(W, H, steps, genes):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W + H + steps, n_models=40,
                                              steps=steps, W=W, H=H, genes=genes,
                                              links=(1, 3 * genes[1]), n_exp=2)
    # Every fourth model: no production and no diffusion; its states decay
    # (deg > 0) or, in the second experiment (all inputs 0), never change.
    init[1] = 0.0
    still = np.zeros(batch.n_models, bool)
    still[::4] = True
    rows = np.repeat(still, np.diff(batch.product_offsets))
    batch.products["lim"][rows] = 0.0
    batch.products["dif"][rows] = 0.0
    out = {}
    for sched, cluster in ((grn.SCHEDULE_FIXED_ITEMS, 0), (grn.SCHEDULE_WALK_ITEMS, 0),
                           (grn.SCHEDULE_CLUSTER, 2)):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, cluster_size=cluster)
            raw, states = ev.evaluate_states(batch, max_planes=16)
            _, _, st = ev.evaluate_batch(batch)
        assert st["schedule"] == sched
        out[sched] = (raw, states, st["total_steps"])
    raw, states, total = out[grn.SCHEDULE_WALK_ITEMS]
    assert total <= 40 * 2 * steps and (steps == 1 or total < 40 * 2 * steps)
    f_raw, f_states, f_total = out[grn.SCHEDULE_FIXED_ITEMS]
    assert np.array_equal(f_states, states) and np.array_equal(f_raw, raw) and f_total == total
    c_raw, c_states, c_total = out[grn.SCHEDULE_CLUSTER]
    assert np.array_equal(c_states, states) and np.array_equal(c_raw, raw) and c_total == total
