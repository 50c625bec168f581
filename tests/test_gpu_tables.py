"""Ray tables made on the device: every form of points against the oracle on the same points
(hits exact, p(d|lambda) within 1e-6 as in the other parity tests). Sizes around the buckets'
and the device's limits, seeds at the ends of [0, 1) and outside it (the host's table), each
size twice (the first call sorts, the second has the size's order); the caller's own points
in any order, equal, clustered (too many for a bucket: the host's table) or outside (0, 1)."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import precision as P
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def design():
    return synth.random_design(np.random.default_rng(12), 3, 48)[:2]


@pytest.fixture(scope="module")
def ctx():
    c = cpd.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("R", [1, 2, 32, 33, 1023, 1024, 1025, 2049, 16384, 16385])
@pytest.mark.parametrize("seeds", [[0.0], [0.5], [1e-17], [1.0 - 2.0 ** -53], [0.123, 0.9], [-0.3], [1.75]],
                         ids=lambda s: "_".join(str(v) for v in s))
def test_seeded_tables(design, ctx, R, seeds):
    spec, d = design
    for adaptive in (False, True):
        for call in range(2):
            f = spec.gpu_fitness_full(seeds, max_n=20, max_eval=R, adaptive=adaptive, context=ctx)
            hits = 0
            for s in seeds[: f.wavelengths // 20]:
                lam, rays = O.gpu_points(s, 20), O.gpu_points(s, R, 1)
                st = (O.fitness_adaptive_points if adaptive else O.fitness_points)(d, lam, rays)[1]
                hits += st["hits"]
            assert f.hits == hits, (adaptive, call)


def _points(kind, R):
    rng = np.random.default_rng(R)
    if kind == "uniform":
        return rng.uniform(size=R)
    if kind == "equal":
        return np.full(R, 0.37)
    if kind == "pairs":
        return np.repeat(rng.uniform(size=R // 2 + 1), 2)[:R]
    if kind == "clustered":
        return 0.5 + 1e-9 * rng.uniform(size=R)
    if kind == "descending":
        return np.linspace(1.0, 0.0, R + 2)[1:-1]
    if kind == "extreme":
        return np.concatenate([[5e-324, 1e-300, 1e-20, 1.0 - 2.0 ** -53], rng.uniform(size=R)])[:R]
    return np.concatenate([[0.0, 1.0, -0.5, 2.0], rng.uniform(size=R)])[:R]  # outside


@pytest.mark.parametrize("kind", ["uniform", "equal", "pairs", "clustered", "descending", "extreme", "outside"])
@pytest.mark.parametrize("R", [4, 33, 1000, 1025, 16384])
def test_own_points(design, ctx, kind, R):
    spec, d = design
    lam, rays = P.synth_points(0.2, 24), _points(kind, R)
    for mode in (cpd.TRACE_HYBRID, cpd.TRACE_HYBRID | cpd.SAMPLING_ADAPTIVE):
        f, p = spec.gpu_fitness_points(lam, rays, want_p=True, mode=mode, context=ctx)
        po, st = (O.fitness_points if mode == cpd.TRACE_HYBRID else O.fitness_adaptive_points)(d, lam, rays)[:2]
        assert f.hits == st["hits"] and np.abs(p - po).max() <= 1e-6, mode
