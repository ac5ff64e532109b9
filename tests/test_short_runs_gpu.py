"""Batches of a few steps take a launch per step, from four (five at up to 2,048 spins) on one launch: the same bits."""
import numpy as np
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,least", [((300, 64), 5), ((2048,), 5), ((2049, 130), 4)])
@pytest.mark.parametrize("jmax", [1, 9])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5])
def test_short_batches(sizes, least, jmax, steps):
    probs = [sb.Problem.random(n, 0.5, jmax, 0, seed=n) for n in sizes]
    prm = sb.Params.default(sb.DSB, steps=steps, replicas=40, seed=3, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    batch = ctx.batch(probs, prm, want_state=True)
    try:
        for _ in range(2):  # the second run replays what the first one captured
            res = batch.run(seed=3)
            for k, (prob, r) in enumerate(zip(probs, res)):
                prm.seed = 3 + k
                one = ctx.solve(prob, prm, want_state=True)
                assert r.steps_per_launch == (steps if steps >= least else 1) and r.energy_check_ok
                np.testing.assert_array_equal(r.final_x, one.final_x)
                np.testing.assert_array_equal(r.final_y, one.final_y)
                np.testing.assert_array_equal(r.replica_energies, one.replica_energies)
    finally:
        batch.close()
        ctx.close()
