"""Adaptive sampling of a coated design at the rows per SM and rounds where its blocks' warps change
(16, 8, 4, and one warp per row): a design's result is the one it has in a pass of many rows."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 33, 1024, 1025, 3000])
@pytest.mark.parametrize("W", [303, 304, 607, 608, 1215, 1216])
def test_single_call_equals_its_place_in_a_batch(W, R):
    rng = np.random.default_rng([W, R])
    specs = [synth.random_design(rng, int(rng.integers(1, 6)), B)[0] for B in (16, 236)]
    many = cpd.fitness_batch(specs, seeds=0.3, max_n=[W, 2048], max_eval=R,
                             mode=cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE)
    wide = cpd.fitness_batch(specs, seeds=0.3, max_n=[2048, W], max_eval=R,
                             mode=cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE)
    for spec, f in ((specs[0], many[0]), (specs[1], wide[1])):
        g = spec.gpu_fitness_full([0.3], max_n=W, max_eval=R, adaptive=True)
        for k in FIELDS + ("status",):
            assert getattr(f, k) == getattr(g, k), k
