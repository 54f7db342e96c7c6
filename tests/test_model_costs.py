"""grn_model_costs follows the kernel's own weights: 13 per gene in use, and 5
plus 5 per link where it is regulated, counted from the compiled program."""
import re

import numpy as np

import grn_b200 as grn
import synth


def test_costs_count_genes_and_links():
    _, batch, _, _ = synth.workload("uneven_64x64", seed=2, n_models=200)
    batch.links["hill_coef"][::7] = 0.0
    batch.links["hill_coef"][1::5] *= -1.0  # some genes lose their last activator
    costs = grn.model_costs(batch, 2)
    for m in range(batch.n_models):
        text = grn.describe_model(*batch.model(m), 2)
        links = [int(a) + int(b) for a, b in re.findall(r"or (\d+) and (\d+)", text)]
        assert costs[m] == sum(13 + (5 + 5 * n if n else 0) for n in links), text
    assert len(np.unique(costs)) > 20
