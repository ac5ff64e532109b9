"""aSB on both sides of the lines between its forms (clusters, a launch per step on rows or on register tiles, with and
without a trace): a replica's trajectory has the same bits in all of them, and beside any number of others."""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,traced", [
    (64, 9, 1), (65, 9, 1),                    # tiles up to 64 spins with a trace
    (512, 28, 0), (512, 29, 0),                # two rounds of clusters, then a launch per step
    (300, 120, 0), (300, 121, 0),              # 570 and 608 row-per-warp CTAs
    (400, 64, 1), (400, 57, 1), (512, 49, 1),  # 400 of them with a trace
    (513, 56, 0), (513, 57, 0), (513, 39, 1), (513, 40, 1),
    (640, 23, 0), (640, 24, 0), (640, 8, 0), (899, 8, 1), (900, 8, 1),
    (1399, 12, 0), (1400, 12, 0),
])
def test_forms_have_the_same_bits(n, R, traced):
    prob = sb.Problem.from_dense(instances.complete_pm1(n, seed=3))
    out = []
    for replicas in (3, R):
        ctx = sb.Context(0)
        try:
            prm = sb.Params.default(sb.ASB, steps=9, replicas=replicas, init_mode=sb.INIT_REFERENCE, trace=traced, trace_all=traced)
            out.append(ctx.solve(prob, prm, want_state=True))
        finally:
            ctx.close()
    np.testing.assert_array_equal(out[0].final_x.view(np.uint32), out[1].final_x[:3].view(np.uint32))
    np.testing.assert_array_equal(out[0].final_y.view(np.uint32), out[1].final_y[:3].view(np.uint32))
    np.testing.assert_array_equal(out[0].replica_energies, out[1].replica_energies[:3])
    if traced:
        np.testing.assert_array_equal(out[0].energy_trace_all, out[1].energy_trace_all[:, :3])
    assert out[1].energy_check_ok
