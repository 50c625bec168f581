"""transmission_probability where the coated exit face is met at both sides of cos 0.5 (glass of an
index near 1, a steep exit face): rays of one wavelength hit with more than one transmittance, and
the wavelength is left to the general kernel. Equal to the oracle, all such wavelengths in one more
launch, whose time counts."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import synth, workload

pytestmark = pytest.mark.gpu


def _two_sided(rng, B):
    """A design whose rays meet the exit face on both sides of cos 0.5 and reach the detector."""
    lam, u = np.full(64, 0.66), np.linspace(0.02, 0.98, 64)
    while True:
        d = workload.draw_params(rng, 1, B, curvature=float(rng.uniform(0.05, 0.4)))
        n = float(rng.uniform(1.02, 1.14))
        d.update(glasses=[[0.0, 0.0, 0.0, 0.0, -0.02, n]], angles=[float(rng.uniform(-0.3, 0.3)), float(rng.uniform(0.9, 1.15))],
                 det_angle=float(rng.uniform(-1.2, 1.2)))
        d = O.accept_params(d)
        if d is None:
            continue
        bins, ts = O.trace_pairs(d, (lam - 0.5) / 0.32, u)
        hit = bins < B
        if hit.sum() >= 20 and np.ptp(ts[hit]) > 1e-3:
            return synth.spectrometer_from_dict(d), d


@pytest.mark.parametrize("B,n,max_m", [(8, 1, 3000), (16, 40, 4096), (300, 33, 1024)])
def test_handed_back_wavelengths(B, n, max_m):
    rng = np.random.default_rng(B)
    for _ in range(2):
        spec, d = _two_sided(rng, B)
        w = 0.66 + 0.32 * (np.arange(n) - (n - 1) / 2) / n
        ctx = cpd.Context(0)
        p, rays = spec.transmission_probability(w, max_m=max_m, return_rays=True, context=ctx)
        po, ro = zip(*(O.p_dets_l_wavelength_count(d, x, max_m) for x in w))
        assert np.array_equal(rays, np.array(ro)) and np.array_equal(p, np.array(po))
        ms, launches = ctx.last_timing()
        assert launches == 3 and ms > 0.0
        ctx.close()
