"""The bounded waits of steps without a block barrier.  A count that never
comes (test hook): the warps that wait for it give up together, the block or
the whole cluster leaves, the call reports it within seconds, and the same
context then gives the right result.  Runs whose counts could overflow keep the
barrier (CPU, over the kernel's own header)."""
import os
import subprocess
import time

import numpy as np
import pytest

import grn_b200 as grn
import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_runs_whose_counts_could_overflow(tmp_path):
    exe = str(tmp_path / "chunk_counts")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(CUDA_HOME, "include"),
                    os.path.join(ROOT, "tests", "cpp", "chunk_counts.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,sched,cluster", [
    (64, 64, grn.SCHEDULE_FIXED_ITEMS, 0),   # 16 chunks, waits of both neighbours
    (8, 8, grn.SCHEDULE_FIXED_ITEMS, 0),     # one chunk, which waits for its own parts
    (100, 40, grn.SCHEDULE_CLUSTER, 2),      # the other CTA learns by its halo counts
    (64, 64, grn.SCHEDULE_CLUSTER, 8),
])
def test_a_missing_count_is_reported(W, H, sched, cluster):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W + H, n_models=3, steps=40,
                                              W=W, H=H, genes=(2, 6))
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(sched, cluster_size=cluster)
        _, want, _ = ev.evaluate_batch(batch)
        ev.set_test_hooks(grn.TEST_WITHHOLD_CHUNK_COUNT)
        t0 = time.perf_counter()
        with pytest.raises(grn.GrnError) as e:
            ev.evaluate_batch(batch)
        # Three models at a time, a give-up of about a second each.
        assert time.perf_counter() - t0 < 30
        assert e.value.status == 10 and "neighbouring warp" in str(e.value)
        ev.set_test_hooks(0)
        _, raw, st = ev.evaluate_batch(batch)
        assert st["schedule"] == sched
    assert np.isfinite(raw).all()
    np.testing.assert_array_equal(raw, want)


@pytest.mark.gpu
def test_the_hook_leaves_barrier_steps_alone():
    """Models with an early-exit threshold pass a barrier and wait for no count."""
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=5, n_models=3, steps=40)
    params["min_conc_change"] = 1e-6
    with grn.Evaluator(params) as ev:
        ev.set_experiments(init, tgt)
        ev.set_schedule(grn.SCHEDULE_FIXED_ITEMS)
        _, want, _ = ev.evaluate_batch(batch)
        ev.set_test_hooks(grn.TEST_WITHHOLD_CHUNK_COUNT)
        _, raw, _ = ev.evaluate_batch(batch)
    np.testing.assert_array_equal(raw, want)
