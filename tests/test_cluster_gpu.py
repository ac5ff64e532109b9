"""Plain FP32 solves of up to 512 spins in one launch of clusters (aSB, bSB, dSB with couplings the bit planes do not
take, NMFA) against one launch per step (SB_PLAIN_PERSIST=0), bit for bit: the same sums in the same order.

Sizes sit on the edges of the 32-row CTAs, the two rows of a warp, the float4 groups of a lane and the rule.
"""
import numpy as np
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu


def _problem(n, fields, seed=0):
    rng = np.random.default_rng(n + seed)
    J = np.triu(rng.normal(size=(n, n)) / np.sqrt(n), 1).astype(np.float32)
    h = (0.1 * rng.normal(size=n)).astype(np.float32) if fields else None
    return sb.Problem.from_dense(J + J.T, h)


def _both(run, monkeypatch):
    out = []
    for value in (None, "0"):
        if value is None:
            monkeypatch.delenv("SB_PLAIN_PERSIST", raising=False)
        else:
            monkeypatch.setenv("SB_PLAIN_PERSIST", value)
        ctx = sb.Context(0)
        try:
            out.append(run(ctx))
        finally:
            ctx.close()
    return out


@pytest.mark.parametrize("variant", [sb.ASB, sb.BSB, sb.DSB])
@pytest.mark.parametrize("n,R,steps,fields,one", [
    (1, 2, 3, True, True),
    (2, 1, 1, False, True),
    (31, 3, 2, True, True),
    (33, 5, 25, False, True),      # a second CTA of one row
    (64, 8, 24, True, True),       # whole CTAs
    (127, 1, 25, False, True),
    (129, 12, 20, True, True),     # a second float4 group of one column
    (257, 20, 15, True, True),     # nine CTAs: more than a portable cluster
    (383, 4, 20, False, True),
    (512, 2, 25, True, True),      # sixteen CTAs
    (512, 39, 6, False, False),    # more CTAs than the rule takes
    (513, 1, 10, True, True),      # the exchange through L2
])
def test_cluster_solve_equals_per_step(variant, n, R, steps, fields, one, monkeypatch):
    if variant == sb.ASB:
        fields = False
    prob = _problem(n, fields)
    prm = sb.Params.default(variant, steps=steps, replicas=R, seed=9, field_mode=sb.FIELD_FP32)
    a, b = _both(lambda ctx: ctx.solve(prob, prm, want_state=True), monkeypatch)
    assert b.steps_per_launch == 1 and a.steps_per_launch == (steps if one else 1)
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
    np.testing.assert_array_equal(a.best_spins, b.best_spins)


@pytest.mark.parametrize("n,R,stages", [(1, 1, 2), (33, 4, 5), (100, 31, 20), (257, 3, 10), (512, 2, 1), (300, 90, 3)])
def test_cluster_nmfa_equals_per_sweep(n, R, stages, monkeypatch):
    prob = _problem(n, False, 7)
    prm = sb.NmfaParams.default(samples=R, stages=stages, seed=5, field_mode=sb.FIELD_FP32)
    a, b = _both(lambda ctx: ctx.nmfa_solve(prob, prm, want_states=True), monkeypatch)
    np.testing.assert_array_equal(a.states, b.states)
    np.testing.assert_array_equal(a.samples, b.samples)
