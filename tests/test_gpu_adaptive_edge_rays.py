"""Adaptive sampling of rows with more rays at a bin's edge than a block lists (or such rays only
past the row's stop), and of rows whose hits have more than one transmittance: rays, hits and
p(d|lambda) are those that the same rows have in a pass of many rows, where a warp takes a row round
by round, and the oracle's."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS
from test_gpu_tp_handed_back import _two_sided

pytestmark = pytest.mark.gpu
MODE = cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE


def _edge_and_middle(spec, d, lam, B):
    """Two ray points at wavelength lam: one on the upper edge of a bin, one well inside that bin."""
    (px, py), (ux, uy) = spec.design.det_position, spec.design.det_direction

    def pos(u):
        try:
            path = spec.ray_trace(lam, d["beam_y_mean"] - d["beam_width"] * O.norminv(u))
        except cpd.RayTraceError:
            return None
        return float((path[-1][0] - px) * ux + (path[-1][1] - py) * uy)

    us = np.linspace(0.2, 0.8, 400)
    ps = [pos(u) for u in us]
    for q in range(1, B - 1):
        edge, mid = (d["linear_intercept"] + q * d["linear_slope"] + f * d["bin_size"] for f in (1.0, 0.5))
        found = []
        for want in (edge, mid):
            for i in range(len(us) - 1):
                if ps[i] is None or ps[i + 1] is None or (ps[i] - want) * (ps[i + 1] - want) > 0:
                    continue
                lo, hi = us[i], us[i + 1]
                while hi - lo > 1e-15 and lo < (lo + hi) / 2 < hi:
                    m = (lo + hi) / 2
                    if pos(m) is None:
                        break
                    lo, hi = (m, hi) if (pos(m) - want) * (ps[i] - want) > 0 else (lo, m)
                found.append(lo)
                break
        if len(found) == 2 and abs(found[0] - found[1]) > 1e-3:
            return found
    return None


def _cases(B):
    rng = np.random.default_rng(77)
    out = []
    while len(out) < 3:
        spec, d, _ = synth.random_design(rng, 3, B)
        u0 = float(rng.uniform(0.2, 0.8))
        lo, hi = d["wavelength_bounds"]
        got = _edge_and_middle(spec, d, lo + (hi - lo) * u0, B)
        if got:
            k = np.arange(1300)  # the edge ray hits on one side of u0 and is lost on the other
            out.append((spec, d, u0 + 1e-9 * (1 + k // 2) * (-1.0) ** k, *got))
    return out


# few rows of a narrow detector are decided many rounds at once, of a wide one in groups of 16 rounds
@pytest.mark.parametrize("B", [24, 300])
@pytest.mark.parametrize("kind", ["all along", "past the stop", "few"])
def test_rows_alone_equal_rows_among_many(kind, B):
    R = 8192
    for spec, d, lam, edge, middle in _cases(B):
        if kind == "all along":  # half of the rays on the edge
            rays = np.tile([edge, middle], R // 2)
        elif kind == "past the stop":  # every ray of the first rounds hits the one bin
            rays = np.r_[np.full(64, middle), np.full(R - 64, edge)]
        else:  # fewer than the list holds
            rays = np.full(R, middle)
            rays[::100] = edge
            rays[1::3] = 0.999999  # and hits that vary
        f, p = spec.gpu_fitness_points(lam, rays, want_p=True, mode=MODE)
        g, q = spec.gpu_fitness_points(lam[:8], rays, want_p=True, mode=MODE)
        assert np.array_equal(p[:8], q)
        po, st, n = O.fitness_adaptive_points(d, lam[:8], rays, 8)
        assert np.abs(q - po).max() <= 1e-6 and g.rays == int(n.sum()) and g.hits == st["hits"]
        assert (np.sum(n == 32) >= 4) if kind == "past the stop" else np.any(n > 32)


@pytest.mark.parametrize("R", [40, 2000, 8192])
@pytest.mark.parametrize("B", [8, 100, 300])
def test_rows_of_two_transmittances(B, R):
    rng = np.random.default_rng([B, R])
    for _ in range(3):
        spec, d = _two_sided(rng, B)
        lam, rays = rng.uniform(size=1300), rng.uniform(size=R)
        f, p = spec.gpu_fitness_points(lam, rays, want_p=True, mode=MODE)
        for n in (5, 330, 700):  # one row per SM at most, two or three, four or more
            g, q = spec.gpu_fitness_points(lam[:n], rays, want_p=True, mode=MODE)
            assert np.array_equal(p[:n], q)
        po, st, count = O.fitness_adaptive_points(d, lam[:200], rays, 8)
        assert np.abs(p[:200] - po).max() <= 1e-6
        g, _ = spec.gpu_fitness_points(lam[:200], rays, want_p=True, mode=MODE)
        assert g.rays == int(count.sum()) and g.hits == st["hits"]


@pytest.mark.parametrize("W", [5, 60, 400])
def test_both_kinds_of_designs_in_one_pass(W):
    rng = np.random.default_rng(W)
    specs = [_two_sided(rng, 16)[0], synth.random_design(rng, 3, 40, ar_coated=False)[0], synth.random_design(rng, 2, 200)[0]]
    for R in (33, 2000, 9000):
        mixed = cpd.fitness_batch(specs, seeds=0.3, max_n=W, max_eval=R, mode=MODE)
        for spec, f in zip(specs, mixed):
            g = spec.gpu_fitness_full([0.3], max_n=W, max_eval=R, adaptive=True)
            for k in FIELDS + ("status",):
                assert getattr(f, k) == getattr(g, k), (R, k)
