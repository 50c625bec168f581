"""transmission_probability by certified pieces: rays consumed and p(d|lambda) bits equal the
oracle's, over designs that lose rays in every way, budgets around the chunk and the limit of the
tables (beyond it, and without a coating, the general kernel), and detectors of few and many bins.
"""
import numpy as np
import pytest

import oracle as O
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


def _check(spec, d, w, max_m):
    p, rays = spec.transmission_probability(w, max_m=max_m, return_rays=True)
    po, ro = zip(*(O.p_dets_l_wavelength_count(d, x, max_m) for x in w))
    assert np.array_equal(rays, np.array(ro))
    assert np.array_equal(p, np.array(po))


@pytest.mark.parametrize("kw", [{}, {"angle_range": (0.5, 1.3)}, {"beam_width": 6.0}, {"curvature": 0.5},
                                {"ar_coated": False}], ids=["plain", "steep", "wide_beam", "curved", "uncoated"])
@pytest.mark.parametrize("B", [2, 31, 64, 257])
def test_equals_oracle(kw, B):
    rng = np.random.default_rng(B)
    for _ in range(3):
        spec, d, _ = synth.random_design(rng, int(rng.integers(2, 7)), B, max_tries=50000, **kw)
        w = np.concatenate([rng.uniform(0.45, 0.9, 40), [0.2, 1.5]])
        _check(spec, d, w, 4096)


@pytest.mark.parametrize("max_m", [1, 2, 255, 256, 1023, 1024, 1025, 65536, 65537])
def test_budgets(max_m):
    spec, d, _ = synth.random_design(np.random.default_rng(8), 3, 12)
    _check(spec, d, np.linspace(0.4, 1.0, 33), max_m)
