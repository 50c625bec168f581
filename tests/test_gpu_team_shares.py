"""Warps per row of the row kernel where the rule on a half-warp's share turns (64 and 256 rays, for
teams of 2 to 16): every choice gives the ray-by-ray kernels' integers."""
import numpy as np
import pytest

from compound_prism_designer import precision as P
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS, _ray_by_ray

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [60, 150, 300, 700])
@pytest.mark.parametrize("R", [256, 257, 511, 512, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096])
def test_teams_equal_ray_by_ray(W, R):
    spec, _, _ = synth.random_design(np.random.default_rng([W, R]), 4, 60)
    lam_u, ray_u = P.synth_points(0.4, W), P.synth_points(0.1, R, first=1)
    f, p = spec.gpu_fitness_points(lam_u, ray_u, want_p=True)
    g, q = _ray_by_ray(spec, lam_u, ray_u)
    assert np.array_equal(p, q)
    for k in FIELDS:
        assert getattr(f, k) == getattr(g, k), k
