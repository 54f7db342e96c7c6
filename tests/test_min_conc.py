"""Models under a minimum concentration on the fast path against the exact
path, which the no-allocation entry point always takes: the same raw errors
and step counts, with thresholds that clamp few and most cells, inputs below
the threshold (kept where their rate is 0), with and without early exit."""
import numpy as np
import pytest

import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(48, 40), (33, 31), (128, 70)])
@pytest.mark.parametrize("min_conc", [1e-30, 0.01, 0.3])
@pytest.mark.parametrize("threshold", [0.0, 1e-3])
def test_clamped_models_match_the_exact_path(W, H, min_conc, threshold):
    torch = pytest.importorskip("torch")
    params, batch, init, tgt = synth.workload("uneven_64x64", seed=W + H, n_models=24, steps=80,
                                              W=W, H=H, n_exp=2)
    params["min_conc"] = min_conc
    params["min_conc_change"] = threshold
    # Every third model neither produces, decays nor diffuses: its inputs stay.
    rows = np.repeat(np.arange(batch.n_models) % 3 == 0, np.diff(batch.product_offsets))
    for k in ("lim", "deg", "dif"):
        batch.products[k][rows] = 0.0
    n = batch.n_models
    d_me = torch.full((n,), 1000.0, dtype=torch.float64, device="cuda")
    out = []
    for exact in (False, True):
        d_raw = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
        d_steps = torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        if exact:
            d_init = torch.tensor(init, dtype=torch.float32, device="cuda")
            d_tgt = torch.tensor(tgt, dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            grn.evaluate_batch_noalloc(params, 2, d_init.data_ptr(), d_tgt.data_ptr(), batch,
                                       d_me.data_ptr(), d_raw.data_ptr(), d_steps.data_ptr())
            grn.evaluate_batch_noalloc_status()
        else:
            with grn.Evaluator(params) as ev:
                ev.set_experiments(init, tgt)
                pk = ev.pack(batch)
                pk.run(d_me.data_ptr(), d_raw.data_ptr(), d_steps.data_ptr())
                pk.status()
                pk.free()
        out.append((d_raw.cpu().numpy(), d_steps.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
