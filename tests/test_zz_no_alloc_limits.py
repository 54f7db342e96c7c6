"""The no-allocation entry at its limits: grids whose sizes do not fit 32 bits
are refused like others that exceed the scratch; odd heights whose own rows
fill the scratch run, in bounds (the bounds-checked library gives the same).

Run as a script: python tests/test_zz_no_alloc_limits.py LIB W H prints the raw
errors that LIB gives for such a grid."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "grn-gpu-performance_b200"), os.path.join(ROOT, "oracle")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import binding as oracle  # noqa: E402
import grn_b200 as grn  # noqa: E402
import synth  # noqa: E402

pytestmark = pytest.mark.gpu

CHECKED = os.path.join(os.path.dirname(grn.LIB_PATH), "libgrn_b200_checked.so")


def _case(W, H):
    return synth.workload("small_32x32", seed=W, n_models=3, steps=4, W=W, H=H, genes=(3, 3),
                          links=(4, 9))


def _noalloc(params, batch, init, tgt):
    import torch
    n = batch.n_models
    d_init = torch.tensor(init, dtype=torch.float32, device="cuda")
    d_tgt = torch.tensor(tgt, dtype=torch.float32, device="cuda")
    d_me = torch.full((n,), 1000.0, dtype=torch.float64, device="cuda")
    d_raw = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    grn.evaluate_batch_noalloc(params, 1, d_init.data_ptr(), d_tgt.data_ptr(), batch,
                               d_me.data_ptr(), d_raw.data_ptr())
    grn.evaluate_batch_noalloc_status()
    return d_raw.cpu().numpy()


# With a row more per plane the slot would not fit the 64 MiB: the first two fill
# to 94% and 99%, 45 rows to 97%; the others hold planes in shared memory.
@pytest.mark.parametrize("W,H", [(220000, 7), (690000, 1), (44500, 45), (1, 1), (33, 31), (90, 61)])
def test_odd_heights_fill_the_scratch(W, H, built_libs):
    params, batch, init, tgt = _case(W, H)
    raw = _noalloc(params, batch, init, tgt)
    _, want, _ = oracle.evaluate_batch(params, init, tgt, batch, np.full(batch.n_models, 1000.0))
    assert np.abs(raw - want).max() <= 1e-4 * want.max()
    r = subprocess.run([sys.executable, __file__, CHECKED, str(W), str(H)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert np.array_equal(np.array([float.fromhex(v) for v in r.stdout.split()]), raw)


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


if __name__ == "__main__":
    grn.load_library(sys.argv[1])
    print(" ".join(float(v).hex() for v in _noalloc(*_case(int(sys.argv[2]), int(sys.argv[3])))))
