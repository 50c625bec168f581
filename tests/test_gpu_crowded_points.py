"""Own ray points that crowd in the device sort's buckets go to the host's table at once: one upload,
as for points that the device cannot sort at all, and no pass in vain."""
import numpy as np
import pytest

import compound_prism_designer as cpd
import oracle as O
from compound_prism_designer import precision as P
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ar", [True, False])
@pytest.mark.parametrize("R", [33, 64, 1000, 4000, 16384])
@pytest.mark.parametrize("kind", ["equal", "cluster", "a fifth"])
def test_one_pass(kind, R, ar):
    spec, d = synth.random_design(np.random.default_rng(12), 3, 48, ar_coated=ar)[:2]
    rng = np.random.default_rng(R)
    rays = np.full(R, 0.37) if kind == "equal" else 0.5 + 1e-9 * rng.uniform(size=R) if kind == "cluster" else rng.uniform(size=R)
    if kind == "a fifth":
        rays[: R // 5] = 0.3
        rng.shuffle(rays)
    lam = P.synth_points(0.2, 16)
    ctx = cpd.Context(0)
    f, p = spec.gpu_fitness_points(lam, rays, want_p=True, context=ctx)
    up = ctx.last_transfer_bytes()[0]
    po, st = O.fitness_points(d, lam, rays)[:2]
    assert f.hits == st["hits"] and np.abs(p - po).max() <= 1e-6
    if kind != "a fifth" or R >= 1000:  # (a fifth of 64 rays are no more than a bucket holds)
        outside = rays.copy()
        outside[0] = 2.0  # for the host, and lost: its table is a ray shorter (an upload's parts are 256 bytes)
        spec.gpu_fitness_points(lam, outside, context=ctx)
        assert abs(up - ctx.last_transfer_bytes()[0]) <= 256
    ctx.close()
