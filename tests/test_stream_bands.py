"""The streaming schedule's bands without a block barrier between them, against
planes in global memory stepped with one: one band, two, and many, short last
bands, odd heights, more and fewer warps than items, both block sizes, fast and
exact models.  The same bits."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,genes", [
    (64, 6, (2, 4)), (256, 33, (8, 16)), (300, 41, (12, 16)), (256, 21, (16, 16)), (5, 90, (2, 8)),
])
@pytest.mark.parametrize("threshold", [0.0, 1e-2])
def test_bands_match_global_planes(W, H, genes, threshold):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W + H, n_models=6, steps=41,
                                              W=W, H=H, genes=genes, links=(2, 3 * genes[1]),
                                              n_exp=2)
    params["min_conc_change"] = threshold
    batch.links["dis_const"][batch.link_offsets[0]] = 0.0  # model 0 takes the exact path
    out = []
    for sched, threads in ((grn.SCHEDULE_GLOBAL, 0), (grn.SCHEDULE_STREAM, 0),
                           (grn.SCHEDULE_STREAM, 512), (grn.SCHEDULE_STREAM2, 0)):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, threads=threads)
            raw, states = ev.evaluate_states(batch, max_planes=16)
            _, _, st = ev.evaluate_batch(batch)
        assert st["schedule"] == sched
        out.append((raw, states, st["total_steps"]))
    for raw, states, total in out[1:]:
        assert np.array_equal(states, out[0][1], equal_nan=True)
        assert np.array_equal(raw, out[0][0], equal_nan=True) and total == out[0][2]
