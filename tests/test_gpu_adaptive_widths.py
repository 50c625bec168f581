"""Adaptive passes that mix detector widths, with tables of more rounds than a block decides at once:
each design's result is the one it has alone. A narrow detector beside a wider one needs other
shared memory than either alone (tests/test_adapt_layout.py holds the sizes)."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS

pytestmark = pytest.mark.gpu
MODE = cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE


@pytest.mark.parametrize("R", [2049, 8192, 16384])
@pytest.mark.parametrize("widths", [(256, 260), (512, 520, 3), (816, 817), (256, 1024, 40)])
def test_mixed_widths_equal_alone(widths, R):
    rng = np.random.default_rng([*widths, R])
    specs = [synth.random_design(rng, int(rng.integers(1, 6)), B)[0] for B in widths]
    for W in (24, 260):  # one row per SM at most, and several
        mixed = cpd.fitness_batch(specs, seeds=0.3, max_n=W, max_eval=R, mode=MODE)
        for spec, f in zip(specs, mixed):
            g = spec.gpu_fitness_full([0.3], max_n=W, max_eval=R, adaptive=True)
            for k in FIELDS + ("status",):
                assert getattr(f, k) == getattr(g, k), (W, k)
