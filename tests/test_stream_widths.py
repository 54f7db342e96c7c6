"""Forced streaming schedules on the widest grids of which a band of one row fits
shared memory, and just past those: the bits of planes in global memory, and
wider ones refused."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


def _workload(W, H, genes):
    return synth.workload("uneven_64x64", seed=W + genes, n_models=3, steps=9, W=W, H=H,
                          genes=(genes, genes), links=(6 * genes, 6 * genes))  # all in use


@pytest.mark.parametrize("sched,W,genes", [
    (grn.SCHEDULE_STREAM, 1100, 8), (grn.SCHEDULE_STREAM, 1150, 8), (grn.SCHEDULE_STREAM, 1176, 8),
    (grn.SCHEDULE_STREAM, 550, 16), (grn.SCHEDULE_STREAM, 581, 16),
    (grn.SCHEDULE_STREAM2, 830, 8), (grn.SCHEDULE_STREAM2, 880, 8),
])
def test_widest_bands(sched, W, genes):
    params, batch, init, tgt = _workload(W, 11, genes)
    out = []
    for s in (grn.SCHEDULE_GLOBAL, sched):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(s)
            out.append(ev.evaluate_states(batch, max_planes=16))
            assert ev.evaluate_batch(batch)[2]["schedule"] == s
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("sched,W,genes", [
    (grn.SCHEDULE_STREAM, 1200, 8), (grn.SCHEDULE_STREAM, 600, 16), (grn.SCHEDULE_STREAM2, 900, 8),
])
def test_wider_grids_are_refused(sched, W, genes):
    params, batch, init, tgt = _workload(W, 11, genes)
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(sched)
        with pytest.raises(grn.GrnError) as e:
            ev.evaluate_batch(batch)
        assert e.value.status == 6  # GRN_ERR_CAPACITY
