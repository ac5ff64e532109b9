"""Large instances with more than 64 replicas, whose couplings L2 does not hold: on both sides of the lines between 64-replica
items that stream their couplings twice and 128-replica tiles, the same bits."""
import numpy as np
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,jmax", [(7936, 9), (7937, 9), (6656, 100), (6657, 100)])  # 63 MB as E4M3, 90 MB as 16 hi + lo
def test_single_instances(n, jmax):
    prob = sb.Problem.random(n, 0.3, jmax, 0, seed=n)
    out = []
    for R in (40, 200):  # one item of a CTA; two, or 128-replica units
        ctx = sb.Context(0)
        try:
            out.append(ctx.solve(prob, sb.Params.default(sb.DSB, steps=5, replicas=R, seed=1, field_mode=sb.FIELD_TC), want_state=True))
        finally:
            ctx.close()
    np.testing.assert_array_equal(out[0].final_x, out[1].final_x[:40])
    np.testing.assert_array_equal(out[0].final_y, out[1].final_y[:40])
    np.testing.assert_array_equal(out[0].replica_energies, out[1].replica_energies[:40])
    assert out[1].energy_check_ok


@pytest.mark.parametrize("n,R,jmax,wave", [(9700, 100, 9, True), (10112, 100, 9, False), (10112, 100, 1, True),
                                           (10112, 64, 9, True)])
def test_batches_and_served(n, R, jmax, wave):
    """E2M3 couplings of more than 75 MB with 65 to 128 replicas take a launch per step, the others a wave."""
    prob = sb.Problem.random(n, 0.3, jmax, 0, seed=n)
    prm = sb.Params.default(sb.DSB, steps=6, replicas=R, seed=1, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    batch = ctx.batch([prob], prm, want_state=True)
    try:
        a = batch.run(seed=1)[0]
        b = ctx.solve(prob, prm, want_state=True)
        c = ctx.poll(ctx.submit(prob, prm), n, prm, wait_ms=-1)
    finally:
        batch.close()
        ctx.close()
    assert a.steps_per_launch == 1 or wave
    if (n, jmax) != (10112, 1):  # its 158 items are two rounds, and waves are taken there if a trial finds them faster
        assert a.steps_per_launch == (6 if wave else 1)
    if jmax > 4:
        assert c.steps_per_launch == a.steps_per_launch
    np.testing.assert_array_equal(a.final_x, b.final_x)
    for r in (a, c):
        np.testing.assert_array_equal(r.replica_energies, b.replica_energies)
        assert r.energy_check_ok
