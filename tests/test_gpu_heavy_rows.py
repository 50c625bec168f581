"""Rows with many rays for the float-float trace, which rows_kernel gives a whole block in passes of
small teams: passes with designs of which all or some wavelengths have no reference ray, at the
rule's edges, are equal to passes without the rule, field by field."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import precision as P
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS

pytestmark = pytest.mark.gpu
# beams that reach the exit face at its critical angle or past its edge
HEAVY = [
    dict(glasses=[[-2.680324996, 10.021203833, -15.212251733, 11.816369803, -4.780181604, 2.326481828],
                  [-3.755139648, 13.905530052, -20.851073968, 15.936955774, -6.299424877, 2.528945848],
                  [-3.235094129, 12.032058447, -18.142800548, 13.97170514, -5.581044985, 2.665958136]],
         angles=[0.372132746086994, -0.41268716731384736, 0.21434526532776976, -0.4613471474675551],
         curvature=0.0126614508732401, height=24.304123638594902, beam_y_mean=13.706848601427078,
         det_angle=-0.575397899708143, det_position=(43.23896915455557, 33.94614197988958), det_flipped=True),
    dict(glasses=[[-0.641322035, 2.42148605, -3.723126399, 2.939691329, -1.220074162, 1.467824777],
                  [-0.617327052, 2.358249564, -3.680038185, 2.965885934, -1.263416615, 1.863307956]],
         angles=[-0.27715175045051277, 1.1685674437402194, -0.2948834029095734],
         curvature=0.03657878917769682, height=24.815247096601134, beam_y_mean=9.452581509001176,
         det_angle=-0.5751651513022328, det_position=(114.32039496074565, 119.69141668824099), det_flipped=False),
    dict(glasses=[[-0.564426723, 2.156189063, -3.3649841, 2.708945267, -1.155588603, 1.917037638],
                  [-2.076462177, 7.687961614, -11.52594096, 8.807757393, -3.481427346, 1.951934174],
                  [-3.479341013, 12.979037357, -19.648519097, 15.215488881, -6.128369335, 2.779177994]],
         angles=[-0.4906962660323665, 0.2752830617148543, -0.5576919360257852, 0.22430721966800884],
         curvature=0.015103928041724127, height=22.91153342140253, beam_y_mean=14.112340014340331,
         det_angle=0.5800890011494156, det_position=(44.27178771090366, -24.10986874084626), det_flipped=True),
]


def _heavy(i, B):
    h = HEAVY[i]
    return synth.spectrometer_from_dict(dict(
        h, lengths=[0.0] * len(h["glasses"]), width=7.0, ar_coated=True, bin_count=B, bin_size=25.6 / B,
        linear_slope=32.0 / B, linear_intercept=3.2 / B, det_length=32.0, max_incident_angle=np.pi / 4,
        wavelength_bounds=(0.5, 0.82), beam_width=2.0))


@pytest.mark.parametrize("R", [1, 255, 256, 257, 300, 8192])
def test_batch_with_heavy_rows_equals_single_calls(R):
    rng = np.random.default_rng(R)
    specs = [synth.random_design(rng, 2, 64)[0] if i % 6 else _heavy(i // 6 % 3, 32) for i in range(72)]
    W = [int(rng.integers(1, 200)) for _ in specs]
    retraced = 0.0
    for s, w, f in zip(specs, W, cpd.fitness_batch(specs, seeds=0.3, max_n=W, max_eval=R)):
        g = s.gpu_fitness_full([0.3], max_n=w, max_eval=R)
        for k in FIELDS + ("status",):
            assert getattr(f, k) == getattr(g, k), k
        retraced = max(retraced, f.retraced / (w * R))
    assert retraced > 0.5  # some designs' rows were heavy


@pytest.mark.parametrize("which", range(len(HEAVY)))
@pytest.mark.parametrize("W,R", [(1300, 257), (12300, 8192)])
def test_one_design_of_many_rows_equals_its_parts(W, R, which):
    # the parts' teams are whole blocks
    spec = _heavy(which, 32)
    lam_u, ray_u = P.synth_points(0.2, W), P.synth_points(0.7, R, first=1)
    f, p = spec.gpu_fitness_points(lam_u, ray_u, want_p=True)
    parts = [spec.gpu_fitness_points(lam_u[k:k + 100].copy(), ray_u, want_p=True) for k in range(0, W, 100)]
    assert np.array_equal(p, np.concatenate([q for _, q in parts]))
    for k in ("hits", "retraced", "fast_rays"):
        assert getattr(f, k) == sum(getattr(g, k) for g, _ in parts), k
