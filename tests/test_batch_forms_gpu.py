"""Batches of more than 64 replicas whose waves would give CTAs two items: the form that is timed as the faster one, waves or
a launch per step, gives the bits of single solves, for the batch that was timed and for the next of its kind."""
import numpy as np
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu

STEPS = 6


@pytest.mark.parametrize("sizes,R,jmax", [
    ((5000,) * 4, 200, 9),   # a wave each, half of whose second round is empty: a launch per step is the faster form by 1.5
    ((5000,) * 4, 200, 1),
    ((2300, 2100), 530, 9),  # just above the sizes whose waves are taken untimed; a part-filled last replica tile
    ((2500, 200), 4096, 1),  # the large instance takes no wave at all
])
def test_forms(sizes, R, jmax):
    probs = [sb.Problem.random(n, 0.3, jmax, 0, seed=n + k) for k, n in enumerate(sizes)]
    prm = sb.Params.default(sb.DSB, steps=STEPS, replicas=R, seed=1, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    try:
        runs = []
        for _ in range(2):
            batch = ctx.batch(probs, prm, want_state=True)
            runs.append(batch.run(seed=1))
            batch.close()
        for k, prob in enumerate(probs):
            prm.seed, prm.replicas = 1 + k, min(R, 600)  # a single solve takes no more tiles than SMs
            one = ctx.solve(prob, prm, want_state=True)
            for res in runs:
                assert res[k].energy_check_ok and res[k].steps_per_launch in (1, STEPS)
                np.testing.assert_array_equal(res[k].final_x[:600], one.final_x)
                np.testing.assert_array_equal(res[k].replica_energies[:600], one.replica_energies)
        assert [r.steps_per_launch for r in runs[0]] == [r.steps_per_launch for r in runs[1]]
    finally:
        ctx.close()


def test_untimed_choice_is_not_kept():
    """A batch too short to time leaves the choice to the first one that can."""
    probs = [sb.Problem.random(5000, 0.3, 9, 0, seed=k) for k in range(8)]
    ctx = sb.Context(0)
    try:
        out = []
        for steps in (1, 40):
            batch = ctx.batch(probs, sb.Params.default(sb.DSB, steps=steps, replicas=200, field_mode=sb.FIELD_TC))
            out = batch.run()
            batch.close()
        assert all(r.steps_per_launch == 1 and r.energy_check_ok for r in out)  # 80 us per step where waves take 144
    finally:
        ctx.close()


@pytest.mark.parametrize("sizes,R,jmax", [
    ((1900,) * 7, 400, 9),          # 15 items a tile, 7 tiles an instance, 20 tiles a wave
    ((1000, 1000, 990), 1300, 1),   # 21 tiles of 8 items, 38 tiles a wave: the second instance is in both
])
def test_instances_split_over_waves(sizes, R, jmax):
    probs = [sb.Problem.random(n, 0.3, jmax, 0, seed=n + k) for k, n in enumerate(sizes)]
    prm = sb.Params.default(sb.DSB, steps=20, replicas=R, seed=1, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    try:
        batch = ctx.batch(probs, prm, want_state=True)
        res = batch.run(seed=1)
        batch.close()
        assert all(r.steps_per_launch == 20 for r in res)
        tickets = []
        for k, prob in enumerate(probs):
            prm.seed, prm.replicas = 1 + k, R
            tickets.append(ctx.submit(prob, prm))
        for k, (prob, ticket) in enumerate(zip(probs, tickets)):
            prm.seed, prm.replicas = 1 + k, min(R, 600)
            one = ctx.solve(prob, prm, want_state=True)
            prm.replicas = R
            served = ctx.poll(ticket, prob.n, prm, wait_ms=-1)
            np.testing.assert_array_equal(res[k].final_x[:600], one.final_x)
            np.testing.assert_array_equal(res[k].final_y[:600], one.final_y)
            np.testing.assert_array_equal(res[k].replica_energies[:600], one.replica_energies)
            np.testing.assert_array_equal(served.replica_energies, res[k].replica_energies)
            assert res[k].energy_check_ok and served.energy_check_ok
    finally:
        ctx.close()
