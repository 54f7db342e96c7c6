"""Grids wider than 4096 cells, which only the no-allocation entry takes: the
row of a group by multiplication must equal the integer quotient (CPU, over
the kernel's own header), and fitness must match the FP64 oracle (GPU)."""
import os
import subprocess

import numpy as np
import pytest

import binding as oracle
import grn_b200 as grn
import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
# Around the first widths whose quotient is off by one, far past them, the
# widest and tallest that fit, and the range of the other entry points.
GRIDS = [(33804, 59), (60004, 24), (200000, 8), (200001, 7), (349000, 4), (699000, 1),
         (4096, 4096), (4093, 500), (1, 1000), (2, 3), (4, 4), (5, 77), (64, 64)]


def test_group_rows_equal_integer_division(tmp_path):
    exe = str(tmp_path / "group_rows")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(CUDA_HOME, "include"),
                    os.path.join(ROOT, "tests", "cpp", "group_rows.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe] + [str(v) for g in GRIDS for v in g], capture_output=True,
                         text=True, timeout=120)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(60004, 24), (200000, 8), (33803, 20)])
def test_wide_grids_match_the_oracle(W, H):
    torch = pytest.importorskip("torch")
    params, batch, init, tgt = synth.workload("small_32x32", seed=W, n_models=2, steps=3, W=W,
                                              H=H, genes=(3, 3), links=(4, 9))
    # Only the first and last cells of each row hold anything, in inputs and
    # targets, so a row found one too far shows in the error: a lost group of
    # four cells is 1 / (2 H) of it.
    edge = np.zeros(W, bool)
    edge[:4] = edge[-4:] = True
    init[..., ~edge] = 0.0
    tgt[...] = 0.0
    tgt[..., edge] = np.random.default_rng(W).uniform(0.5, 1.0, tgt[..., edge].shape)
    for m in range(batch.n_models):  # production only where the input is
        rows = slice(batch.product_offsets[m], batch.product_offsets[m + 1])
        batch.products["lim"][rows] = [0.0, 1.0, 1.0]
        batch.products["dif"][rows] = [0.1, 0.0, 0.1]
        links = slice(batch.link_offsets[m], batch.link_offsets[m + 1])
        batch.links["hill_coef"][links] = np.abs(batch.links["hill_coef"][links])
        batch.links["regulator"][links] = 0
        batch.links["is_and"][links] = 0
    d_init = torch.tensor(init, dtype=torch.float32, device="cuda")
    d_tgt = torch.tensor(tgt, dtype=torch.float32, device="cuda")
    d_me = torch.full((2,), 1000.0, dtype=torch.float64, device="cuda")
    d_raw = torch.zeros(2, dtype=torch.float64, device="cuda")
    d_steps = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    grn.evaluate_batch_noalloc(params, 1, d_init.data_ptr(), d_tgt.data_ptr(), batch,
                               d_me.data_ptr(), d_raw.data_ptr(), d_steps.data_ptr())
    grn.evaluate_batch_noalloc_status()
    _, want, steps = oracle.evaluate_batch(params, init, tgt, batch, np.full(2, 1000.0))
    got = d_raw.cpu().numpy()
    assert np.array_equal(d_steps.cpu().numpy(), steps)
    assert (want > 0).all() and np.abs(got - want).max() <= 1e-4 * want.max(), (got, want)
