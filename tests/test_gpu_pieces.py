"""The row kernel of coated designs (certified pieces) against the ray-by-ray kernels, which the
allocation-free entry point runs: the sums of both are the same integers, so every field and
every p(d|lambda) is equal. Sizes at the edges of the split: rows per warp and warps per row,
ranges short enough to go whole to the fast path, one piece's rays and one more, empty warps."""
import ctypes as C

import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import _native as N
from compound_prism_designer import precision as P
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu
FIELDS = ("info", "h_cond", "h_det", "max_sem", "hits", "retraced", "fast_rays", "rays", "wavelengths")


def _ray_by_ray(spec, lam_u, ray_u):
    f = N.Fitness()
    p = np.zeros((lam_u.size, spec.detector_array.bin_count))
    dp = C.POINTER(C.c_double)
    rc = N.lib.cpd_fitness_gpu_points_static(C.byref(spec.design), lam_u.ctypes.data_as(dp), lam_u.size,
                                             ray_u.ctypes.data_as(dp), ray_u.size, cpd.TRACE_HYBRID, C.byref(f),
                                             p.ctypes.data_as(dp))
    assert rc == N.OK, N.status_string(rc)
    return f, p


SIZES = [(1, 1), (1, 4096), (3, 47), (5, 48), (33, 49), (64, 256), (95, 720), (152, 2047), (190, 4096), (380, 1023),
         (381, 1024), (1000, 3001), (1024, 100)]


@pytest.mark.parametrize("W,R", SIZES)
@pytest.mark.parametrize("kw", [{}, {"angle_range": (0.5, 1.3)}, {"beam_width": 6.0}, {"curvature": 0.5}],
                         ids=["plain", "steep", "wide_beam", "curved"])
def test_equals_ray_by_ray(W, R, kw):
    rng = np.random.default_rng([W, R])
    for B in (1, 7, 32, 100, 128):
        spec, _, _ = synth.random_design(rng, int(rng.integers(2, 7)), B, max_tries=50000, **kw)
        lam_u, ray_u = P.synth_points(float(rng.uniform()), W), P.synth_points(float(rng.uniform()), R, first=1)
        f, p = spec.gpu_fitness_points(lam_u, ray_u, want_p=True)
        g, q = _ray_by_ray(spec, lam_u, ray_u)
        assert np.array_equal(p, q), (B, np.abs(p - q).max())
        for k in FIELDS:
            assert getattr(f, k) == getattr(g, k), (B, k, getattr(f, k), getattr(g, k))


@pytest.mark.parametrize("B", [129, 513, 1024])
def test_wide_detector_equals_oracle(B):
    # a row's cells beyond a group's: hits exact, p within 1e-6 (the parity bar of this path)
    spec, d, _ = synth.random_design(np.random.default_rng(B), 3, B)
    lam_u, ray_u = P.synth_points(0.4, 200), P.synth_points(0.4, 3000, first=1)
    f, p = spec.gpu_fitness_points(lam_u, ray_u, want_p=True)
    po, st = O.fitness_points(d, lam_u, ray_u)
    assert f.hits == st["hits"] and np.abs(p - po).max() <= 1e-6


def test_batch_of_many_rows_and_mixed_coatings_equals_single_calls():
    # several rows per warp, groups that end inside a design, and coated and uncoated designs
    # (the ray-by-ray kernels) in one pass
    rng = np.random.default_rng(5)
    specs, W = [], []
    for i in range(40):
        specs.append(synth.random_design(rng, int(rng.integers(1, 7)), int(rng.choice([9, 16, 64, 128, 700])),
                                         ar_coated=i % 4 != 1)[0])
        W.append(int(rng.integers(1, 1200)))
    got = cpd.fitness_batch(specs, seeds=0.3, max_n=W, max_eval=500)
    for s, w, f in zip(specs, W, got):
        g = s.gpu_fitness_full([0.3], max_n=w, max_eval=500)
        for k in FIELDS + ("status",):
            assert getattr(f, k) == getattr(g, k), k
