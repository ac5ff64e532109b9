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
