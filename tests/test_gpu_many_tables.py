"""A batch in which each of more than 65,535 designs has a seed, and so a ray table, of its own."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ar", [True, False])
def test_a_table_per_design(ar):
    spec = synth.random_design(np.random.default_rng(9), 2, 8, ar_coated=ar)[0]
    n = 65_600
    seeds = np.random.default_rng(1).uniform(size=n)
    ctx = cpd.Context(0)
    for _ in range(2):  # sorted by the device; from the kept order
        out = cpd.fitness_batch([spec] * n, seeds=seeds, max_n=2, max_eval=40, context=ctx)
        for i in (0, 1, 32_768, 65_534, 65_535, 65_536, n - 1):
            f = spec.gpu_fitness_full([seeds[i]], max_n=2, max_eval=40)
            assert (out[i].hits, out[i].info) == (f.hits, f.info), i
    ctx.close()
