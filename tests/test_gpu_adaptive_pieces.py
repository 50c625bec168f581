"""Adaptive sampling by certified pieces, in its three forms (a block per row, a warp per row, and
both beside designs without pieces in one pass): rays consumed and hits equal the oracle's, p
within 1e-6, as for the general forms."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import precision as P
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu
MODE = cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE


@pytest.mark.parametrize("B", [1, 3, 64, 129, 513, 1024])
@pytest.mark.parametrize("W,R", [(2, 1), (7, 33), (20, 1000), (12, 8193), (400, 70), (1300, 200)])
def test_equals_oracle(B, W, R):
    spec, d, _ = synth.random_design(np.random.default_rng([B, R]), 2 + B % 4, B)
    lam, rays = P.synth_points(0.3, W), P.synth_points(0.6, R, first=1)
    f, p = spec.gpu_fitness_points(lam, rays, want_p=True, mode=MODE)
    po, st, n = O.fitness_adaptive_points(d, lam, rays, 8)
    assert f.hits == st["hits"] and f.rays == int(n.sum())
    assert np.abs(p - po).max() <= 1e-6


@pytest.mark.parametrize("n", [3, 12])
def test_mixed_pass_equals_alone(n):
    # few rows and many; a pass with designs without pieces takes the same rows by the same forms
    rng = np.random.default_rng(n)
    specs = [synth.random_design(rng, 3, 40, ar_coated=i % 3 != 1)[0] for i in range(n)]
    W = [60] * n if n == 3 else [150] * n
    mix = cpd.fitness_batch(specs, seeds=0.4, max_n=W, max_eval=3000, mode=MODE)
    for s, w, f in zip(specs, W, mix):
        one = cpd.fitness_batch([s], seeds=0.4, max_n=w, max_eval=3000, mode=MODE)[0]
        for k in ("info", "h_cond", "h_det", "max_sem", "rays", "hits", "status"):
            assert getattr(f, k) == getattr(one, k), k
