"""Passes that are run again with the host's ray tables: a seed with a point that rounds to 0 (its
start height is not finite, which the device's table cannot hold). What the passes before it and the
run itself count is counted once: hits, rays consumed and re-traced rays of several seeds, against
the oracle and against the seeds' own calls."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu
ALPHA = 1.0 / 1.61803398874989484820458683436563
ZERO = 1.0 - ALPHA  # its first point is fract(ALPHA + ZERO) = 0


def _designs(ar):
    rng = np.random.default_rng(40 + ar)
    return [synth.random_design(rng, 2 + i, 24, ar_coated=bool(ar))[:2] for i in range(3)]


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("ar", [0, 1])
def test_counts_of_seeds(ar, adaptive):
    assert float(O.gpu_points(ZERO, 1, 1)[0]) == 0.0
    W, R = 7, 100  # few wavelengths: hardly a design converges before its last seed
    all_seeds = 0
    for spec, d in _designs(ar):
        for seeds in ([0.3, ZERO], [0.3, 0.7, ZERO], [ZERO, 0.3], [ZERO]):
            ctx = cpd.Context(0)  # (a context makes such a seed's table on the host from its second use on)
            f = spec.gpu_fitness_full(seeds, max_n=W, max_eval=R, adaptive=adaptive, context=ctx)
            hits = rays = retraced = 0
            for s in seeds[: f.wavelengths // W]:
                lam, u = O.gpu_points(s, W), O.gpu_points(s, R, 1)
                if adaptive:
                    _, st, n = O.fitness_adaptive_points(d, lam, u, 8)
                    rays += int(n.sum())
                else:
                    st = O.fitness_points(d, lam, u)[1]
                    rays += W * R
                hits += st["hits"]
                retraced += spec.gpu_fitness_full([s], max_n=W, max_eval=R, adaptive=adaptive, context=ctx).retraced
            all_seeds += len(seeds) > 1 and f.wavelengths == W * len(seeds)
            assert (f.hits, f.rays, f.retraced) == (hits, rays, retraced), seeds
            ctx.close()
    assert all_seeds >= 3


@pytest.mark.parametrize("adaptive", [False, True])
def test_server_request_with_such_a_seed(adaptive):
    mode = cpd.TRACE_HYBRID | (cpd.SAMPLING_ADAPTIVE if adaptive else 0)
    specs = [s for ar in (0, 1) for s, _ in _designs(ar)]
    ctx = cpd.Context(0)
    sv = cpd.Server(context=ctx)
    for seeds in ([ZERO] * 6, [0.3, ZERO, 0.4, 0.5, ZERO, 0.6]):
        rid = sv.submit([s.design for s in specs], seeds=seeds, max_n=40, max_eval=300, mode=mode)
        out = sv.wait(rid)[0]
        for spec, s, o in zip(specs, seeds, out):
            f = spec.gpu_fitness_full([s], max_n=40, max_eval=300, adaptive=adaptive)
            assert (int(o["hits"]), int(o["rays"]), float(o["info"])) == (f.hits, f.rays, f.info)
    sv.close()
    ctx.close()


def test_server_whose_queue_is_at_its_limit():
    # 17 M rays in f64 take the slot's queue to its largest size; such a seed is still served after it
    (spec, _), = _designs(1)[:1]
    ctx = cpd.Context(0)
    with cpd.Server(slots=1, context=ctx) as sv:
        sv.wait(sv.submit([spec], seeds=0.3, max_n=4096, max_eval=4200, mode=cpd.TRACE_FP64))
        out = sv.wait(sv.submit([spec], seeds=ZERO, max_n=40, max_eval=300))[0]
    f = spec.gpu_fitness_full([ZERO], max_n=40, max_eval=300)
    assert (int(out["hits"][0]), float(out["info"][0])) == (f.hits, f.info)
    ctx.close()
