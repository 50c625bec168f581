"""The device time of single-design calls: by the kernels' own stamps at a context's first
last_timing, by events from then on; the results are the same."""
import time

import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import precision as P
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ar", [True, False])
@pytest.mark.parametrize("kind", ["fixed", "adaptive", "points", "fp64"])
def test_last_timing_before_and_after_it_is_asked_for(kind, ar):
    spec = synth.random_design(np.random.default_rng(3), 3, 32, ar_coated=ar)[0]
    ctx = cpd.Context(0)
    lam, ray = P.synth_points(0.2, 300), P.synth_points(0.7, 2000, first=1)

    def call():
        if kind in ("points", "fp64"):
            return spec.gpu_fitness_points(lam, ray, mode=cpd.TRACE_FP64 if kind == "fp64" else cpd.TRACE_HYBRID,
                                           context=ctx)[0]
        return spec.gpu_fitness_full([0.3], max_n=300, max_eval=2000, adaptive=kind == "adaptive", context=ctx)

    seen = []
    for _ in range(3):
        for _ in range(2):
            t = time.perf_counter()
            f = call()
            wall = (time.perf_counter() - t) * 1e3
        ms, launches = ctx.last_timing()
        assert 0.0 < ms < wall and launches >= 2
        seen.append((f.info, f.hits, launches))
    assert seen[0] == seen[1] == seen[2]
