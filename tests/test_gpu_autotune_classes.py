"""The launch-shape autotuner beside designs that have no shape to tune (coated ones): they neither
take the tuning from the others of their class, nor change the caller's shape."""
import numpy as np
import pytest

import compound_prism_designer as cpd
from compound_prism_designer import synth

pytestmark = pytest.mark.gpu


def _specs(ar, n=6):
    rng = np.random.default_rng(n)
    return [synth.random_design(rng, 3, 32, ar_coated=ar)[0] for _ in range(n)]


@pytest.mark.parametrize("n", [1, 6])
def test_a_coated_batch_leaves_its_class_untuned(n):
    ctx = cpd.Context(0)
    ctx.set_autotune(True)

    def uploads(specs):
        if n == 1:
            specs[0].gpu_fitness_full([0.4], max_n=200, max_eval=512, context=ctx)
        else:
            cpd.fitness_batch(specs, max_n=200, max_eval=512, context=ctx)
        return ctx.last_transfer_bytes()[0]

    coated, uncoated = _specs(True, n), _specs(False, n)
    uploads(coated)
    first, second = uploads(uncoated), uploads(uncoated)
    assert first > 20 * second  # the first call times the candidates, three passes each
    ctx.close()


def test_a_coated_batch_keeps_the_callers_shape():
    ctx = cpd.Context(0)
    ctx.set_launch_shape(64, 4)
    rt, w, ms = cpd.autotune_batch(_specs(True), max_n=200, max_eval=512, context=ctx)
    assert (rt, w) == ctx.launch_shape() == (64, 4) and ms > 0
    ctx.close()
