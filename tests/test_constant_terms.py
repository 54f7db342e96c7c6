"""Links with a Hill coefficient of 0 (the constant Hill value 1/2) with the fast
update against the exact path, which the no-allocation entry always takes: the
same raw errors and step counts on every schedule, with such links alone,
first, last and in the middle of a gene's OR and AND links, as +0 and -0."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


def _batch(W, H, threshold):
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W * 3 + H, n_models=24,
                                              steps=60, W=W, H=H, genes=(2, 6), links=(2, 18),
                                              n_exp=2)
    params["min_conc_change"] = threshold
    for m in range(batch.n_models):
        a, b = batch.link_offsets[m], batch.link_offsets[m + 1]
        hill = batch.links["hill_coef"][a:b]
        if m % 4 == 0:
            hill[0] = 0.0
        elif m % 4 == 1:
            hill[-1] = -0.0
        elif m % 4 == 2:
            hill[::3] = 0.0
        elif m % 8 == 3:
            hill[:] = 0.0  # nothing but constants
    return params, batch, init, tgt


@pytest.mark.parametrize("W,H", [(48, 40), (33, 31)])
@pytest.mark.parametrize("threshold", [0.0, 1e-3])
@pytest.mark.parametrize("min_conc", [0.0, 0.01])
def test_constant_terms_match_the_exact_path(W, H, threshold, min_conc):
    torch = pytest.importorskip("torch")
    params, batch, init, tgt = _batch(W, H, threshold)
    params["min_conc"] = min_conc
    n = batch.n_models
    d_me = torch.full((n,), 1000.0, dtype=torch.float64, device="cuda")
    d_raw = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    d_steps = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_init = torch.tensor(init, dtype=torch.float32, device="cuda")
    d_tgt = torch.tensor(tgt, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    grn.evaluate_batch_noalloc(params, 2, d_init.data_ptr(), d_tgt.data_ptr(), batch,
                               d_me.data_ptr(), d_raw.data_ptr(), d_steps.data_ptr())
    grn.evaluate_batch_noalloc_status()
    want, steps = d_raw.cpu().numpy(), d_steps.cpu().numpy()
    for sched, cluster in ((grn.SCHEDULE_FIXED_ITEMS, 0), (grn.SCHEDULE_WALK_ITEMS, 0),
                           (grn.SCHEDULE_GLOBAL, 0), (grn.SCHEDULE_CLUSTER, 2),
                           (grn.SCHEDULE_STREAM, 0), (grn.SCHEDULE_STREAM2, 0)):
        with grn.Evaluator(params) as ev:
            ev.set_experiments(init, tgt)
            ev.set_schedule(sched, cluster_size=cluster)
            pk = ev.pack(batch)
            pk.run(d_me.data_ptr(), d_raw.data_ptr(), d_steps.data_ptr())
            pk.status()
            pk.free()
        assert np.array_equal(d_raw.cpu().numpy(), want), sched
        assert np.array_equal(d_steps.cpu().numpy(), steps), sched
