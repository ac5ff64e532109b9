"""steps_per_launch and kernel_launches of batches and served requests tell which form ran."""
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu

STEPS = 150


def _problem(n, jmax, seed):
    return sb.Problem.random(n, 0.5, jmax, seed=seed)


@pytest.mark.parametrize("profile", [0, 1])
def test_batch(profile):
    """Two operand types; 4096 replicas of 700 spins are more items than a wave holds, and the
    tile that is timed as the faster one for that bucket may have no waves at all."""
    ctx = sb.Context(0)
    try:
        for ns, R, waves in (((300, 500, 200), 64, (True, True, True)), ((700, 200), 4096, (False, True))):
            probs = [_problem(n, 9 if n == 500 else 1, n) for n in ns]
            batch = ctx.batch(probs, sb.Params.default(sb.DSB, steps=STEPS, replicas=R, field_mode=sb.FIELD_TC, profile=profile))
            res = batch.run()
            batch.close()
            buckets = len({r.field_dtype for r in res})
            assert buckets == (2 if 500 in ns else 1)
            for r, w in zip(res, waves):
                assert r.energy_check_ok
                if all(waves) or not w or profile:
                    assert r.steps_per_launch == (STEPS if w and not profile else 1)
                else:
                    assert r.steps_per_launch in (1, STEPS)
                if all(waves) and not profile:
                    assert r.kernel_launches < 10 * buckets  # states, a wave, signs, energies, results
                else:
                    assert r.kernel_launches >= STEPS
    finally:
        ctx.close()


def test_served():
    ctx = sb.Context(0)
    try:
        reqs = [(_problem(n, 8, n), sb.Params.default(v, steps=STEPS, replicas=R, field_mode=f))
                for n, R, v, f in ((300, 32, sb.DSB, sb.FIELD_TC), (700, 64, sb.DSB, sb.FIELD_TC), (100, 1, sb.BSB, sb.FIELD_FP32))]
        tickets = [ctx.submit(p, prm) for p, prm in reqs]
        res = [ctx.poll(t, p.n, prm, wait_ms=-1) for t, (p, prm) in zip(tickets, reqs)]
        stats = ctx.serving_stats()
    finally:
        ctx.close()
    for r in res[:2]:  # up to 64 steps a launch, more often when requests arrive between
        assert r.energy_check_ok and 1 < r.steps_per_launch <= 64
        assert -(-STEPS // 64) + 1 <= r.kernel_launches < STEPS
    assert res[2].steps_per_launch == STEPS  # solved alone, in one launch
    assert stats["grouped_launches"] < stats["ticks"]
