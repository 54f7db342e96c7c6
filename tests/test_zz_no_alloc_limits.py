"""The no-allocation entry at its limits: grids whose sizes do not fit 32 bits
are refused like others that exceed the scratch."""
import numpy as np
import pytest

import binding as oracle
import grn_b200 as grn
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [
    (262144, 131072),          # 2^32 strips
    (262145, 131071), (2**31 - 1, 2**31 - 1), (2**31 - 1, 1), (1, 2**31 - 1), (65536, 65536),
    (2097153, 1), (1449, 1448),  # more than 2^21 cells
])
def test_huge_grids_are_refused(W, H):
    torch = pytest.importorskip("torch")
    params, batch, _, _ = synth.workload("uneven_64x64", seed=1, n_models=1, steps=1, W=8, H=8)
    params["dim_x"], params["dim_y"] = W, H
    d = torch.zeros(64, dtype=torch.float64, device="cuda")  # refused before any launch
    with pytest.raises(grn.GrnError) as e:
        grn.evaluate_batch_noalloc(params, 1, d.data_ptr(), d.data_ptr(), batch, d.data_ptr(),
                                   d.data_ptr())
    assert e.value.status == 6 and "GRN_NOALLOC_SCRATCH_BYTES" in str(e.value)
