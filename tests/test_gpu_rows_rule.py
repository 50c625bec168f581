"""The line between rows_kernel and the ray-by-ray kernels for coated designs (rows of a pass, bins,
rays per row): a design's result is the same on both sides of it, alone and in a batch."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth
from test_gpu_pieces import FIELDS

pytestmark = pytest.mark.gpu


def _same(f, g):
    for k in FIELDS + ("status",):
        assert getattr(f, k) == getattr(g, k), k


@pytest.mark.parametrize("R", [1, 64, 256, 257])
@pytest.mark.parametrize("W", [8191, 8192])
@pytest.mark.parametrize("B", [1, 80, 81])
def test_one_design(B, W, R):
    spec, other = (synth.random_design(np.random.default_rng([B, i]), 2 + i, B)[0] for i in (0, 1))
    f = spec.gpu_fitness_full([0.3], max_n=W, max_eval=R)
    # in passes of two designs, by rows_kernel (below 16384 rows) and, with R <= 256, ray by ray
    for w in (2, 16384):
        _same(f, cpd.fitness_batch([spec, other], seeds=0.3, max_n=[W, w], max_eval=R)[0])


@pytest.mark.parametrize("R", [64, 256, 257])
@pytest.mark.parametrize("rows", [16383, 16384])
def test_batches(rows, R):
    rng = np.random.default_rng([rows, R])
    specs = [synth.random_design(rng, int(rng.integers(1, 7)), int(B))[0] for B in (7, 64, 300, 32)]
    W = [4000, 5000, 6000, rows - 15000]
    params = cpd.fitness_batch(specs, seeds=0.3, max_n=W, max_eval=R)
    for spec, w, f in zip(specs, W, params):
        _same(f, spec.gpu_fitness_full([0.3], max_n=w, max_eval=R))


@pytest.mark.parametrize("W", [511, 512])  # of the coated designs: 8.4 M rays and a few less
def test_beside_uncoated_designs(W):
    rng = np.random.default_rng(W)
    specs = [synth.random_design(rng, 3, B, ar_coated=ar)[0] for B, ar in ((32, True), (64, False), (9, True))]
    n, R = [W, 40, 512], 8192
    for spec, w, f in zip(specs, n, cpd.fitness_batch(specs, seeds=0.3, max_n=n, max_eval=R)):
        _same(f, spec.gpu_fitness_full([0.3], max_n=w, max_eval=R))
