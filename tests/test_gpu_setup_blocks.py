"""The setup of passes with many rows (blocks of 128 rows) against single calls: blocks that hold
the rows of several designs, a last block that is not full, tables past the staging limit."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [100, 2048, 2049])
def test_pass_of_many_rows_equals_single_calls(R):
    rng = np.random.default_rng(R)
    specs = [synth.random_design(rng, int(rng.integers(1, 7)), 32, ar_coated=i % 3 != 0)[0] for i in range(60)]
    W = [int(rng.integers(1, 6000)) if i % 4 else int(rng.integers(1, 40)) for i in range(60)]
    W[1] += max(0, 90_000 - sum(W))  # past 16 warps of rows per SM
    for s, w, f in zip(specs, W, cpd.fitness_batch(specs, seeds=0.6, max_n=W, max_eval=R)):
        g = s.gpu_fitness_full([0.6], max_n=w, max_eval=R)
        for k in FIELDS + ("status",):
            assert getattr(f, k) == getattr(g, k), k
