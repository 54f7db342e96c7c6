"""The step's work items (chunks of 32 strips of 4 x 2 cells, genes dealt to
several warps) at the sizes where they can go wrong: strip counts around a
chunk, odd heights, ragged widths, rows of groups that do and do not fill a
chunk, more warps than work, walked and owned chunks, genes in global slots.
Every block size and schedule must give the same bits; the states agree with
the FP64 oracle within the suite's parity bar (1e-4 relative + 1e-6)."""
import numpy as np
import pytest

import binding as oracle
import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu

FIXED, WALK, GLOBAL = grn.SCHEDULE_FIXED_ITEMS, grn.SCHEDULE_WALK_ITEMS, grn.SCHEDULE_GLOBAL


@pytest.mark.parametrize("W,H,genes", [
    (4, 62, (2, 6)), (4, 64, (2, 6)), (4, 66, (2, 6)),   # 31, 32, 33 strips of one group
    (3, 5, (2, 5)), (31, 33, (2, 8)), (64, 63, (2, 8)),   # ragged, odd heights
    (36, 17, (9, 16)), (132, 9, (2, 8)), (100, 41, (7, 16)), (128, 2, (2, 4)),
])
def test_every_block_size_gives_the_same_states(W, H, genes):
    steps = 25
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W * 131 + H, n_models=10,
                                              steps=steps, W=W, H=H, genes=genes,
                                              links=(2, 3 * genes[1]))
    batch.links["dis_const"][batch.link_offsets[0]] = 0.0  # model 0 takes the exact path
    batch.links["hill_coef"][batch.link_offsets[1]] = 0.0  # model 1 has a constant term
    chunks = -(-(-(-H // 2) * -(-W // 4)) // 32)
    runs = [(WALK, 512), (WALK, 1024), (GLOBAL, 512), (GLOBAL, 1024)]
    for parts in (1, 2, 3, 4):
        if chunks * parts <= 32:
            runs.append((FIXED, 32 * chunks * parts))
    if chunks < 32:
        runs.append((FIXED, 32 * (chunks + 1)))  # a warp without work
    base = None
    for sched, threads in runs:
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, threads=threads)
            raw, states = ev.evaluate_states(batch, max_planes=16)
            _, raw_b, st = ev.evaluate_batch(batch)
        assert (st["schedule"], st["threads_per_block"]) == (sched, threads)
        assert np.array_equal(raw, raw_b, equal_nan=True)
        if base is None:
            base = (raw, states)
            continue
        assert np.array_equal(states, base[1], equal_nan=True), (sched, threads)
        assert np.array_equal(raw, base[0], equal_nan=True), (sched, threads)
    for m in range(batch.n_models):
        pr, li = batch.model(m)
        ref, _, _ = oracle.simulate(params, init[0], pr, li, steps)
        got = base[1][m, 0, :len(ref)].astype(np.float64)
        near = np.abs(got - ref) <= 1e-6 + 1e-4 * np.abs(ref)
        assert (near | (np.isnan(got) & np.isnan(ref))).all(), m  # K = 0 gives NaN cells
