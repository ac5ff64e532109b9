"""Limits of the device's waits. Shorter than a copy takes they count as the least one: solves under a limit of one clock
give what they give under the default, on every tensor-core kernel that runs a solve. Where a wait runs out (a flag or
word left out on the host's request) the call returns SB_ERR_TIMEOUT and the context goes on."""
import time

import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,n,R,jmax,dtype,trace", [
    (sb.DSB, 300, 96, 1, sb.OPERAND_FP4, 0),     # multi-step kernel, J resident
    (sb.DSB, 1400, 40, 9, sb.OPERAND_FP8, 0),    # J streamed
    (sb.DSB, 300, 96, 1, sb.OPERAND_FP4, 1),     # operands exchanged
    (sb.DSB, 300, 96, 100, sb.OPERAND_BF16, 1),
    (sb.BSB, 1000, 128, 0, sb.OPERAND_BF16X2, 0),  # CTA pairs
    (sb.BSB, 300, 40, 0, sb.OPERAND_BF16X2, 0),
])
def test_short_limits_are_raised(variant, n, R, jmax, dtype, trace):
    if jmax:
        J = instances.erdos_renyi(n, 0.5, seed=n, jmax=jmax, allow_zero=True)
        J[0, 1] = J[1, 0] = jmax
    else:
        J = instances.gaussian(n, seed=2)[0]
    prob = sb.Problem.from_dense(J)
    prm = sb.Params.default(variant, steps=12, replicas=R, seed=5, field_mode=sb.FIELD_TC, operand_dtype=dtype, trace=trace)
    ctx = sb.Context(0)
    try:
        want = ctx.solve(prob, prm, want_state=True)
        ctx.set_wait_limit(1)
        got = ctx.solve(prob, prm, want_state=True)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got.final_x, want.final_x)
    np.testing.assert_array_equal(got.final_y, want.final_y)


def _expires(ctx, call, step):
    """call under a short limit, with one announcement of `step` left out."""
    ctx.set_wait_limit(1_000_000)
    ctx.debug_skip_publish(step)
    t0 = time.perf_counter()
    with pytest.raises(sb.SBError) as ei:
        call()
    assert ei.value.status == 7, str(ei.value)
    assert time.perf_counter() - t0 < 0.5
    ctx.set_wait_limit(0)


@pytest.mark.parametrize("ns,R,jmax", [
    ((700, 300, 100), 64, 1),               # E2M1, J resident
    ((1300, 1300, 1300), 64, 12),           # E2M3 rows too long for that
    ((130,) * 200, 32, 9),                  # up to three items of a CTA
    ((1300, 700, 640), 40, (12, 2, 12)),    # two operand types: the second's waves run on
])
def test_a_wave_gives_up(ns, R, jmax):
    jm = jmax if isinstance(jmax, tuple) else (jmax,) * len(ns)
    Js = [instances.erdos_renyi(n, 0.5, seed=k, jmax=j, allow_zero=True) for k, (n, j) in enumerate(zip(ns, jm))]
    for J, j in zip(Js, jm):
        J[0, 1] = J[1, 0] = j
    ctx = sb.Context(0)
    batch = ctx.batch([sb.Problem.from_dense(J) for J in Js],
                      sb.Params.default(sb.DSB, steps=24, replicas=R, seed=3, field_mode=sb.FIELD_TC), want_state=True)
    try:
        want = batch.run()
        _expires(ctx, batch.run, 12)
        got = batch.run()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a.final_x, b.final_x)
            assert a.energy_check_ok
    finally:
        batch.close()
        ctx.close()


@pytest.mark.parametrize("n,M,R", [(200, 16, 2), (700, 48, 4), (4096, 64, 160)])  # one and two slice warps; two replicas a CTA
def test_sqa_gives_up(n, M, R):
    prob = sb.Problem.from_dense(instances.complete_pm1(n, seed=1))
    prm = sb.SqaParams.default(steps=4, trotter=M, replicas=R, seed=2)
    ctx = sb.Context(0)
    try:
        want = ctx.sqa_solve(prob, prm)
        _expires(ctx, lambda: ctx.sqa_solve(prob, prm), 2)
        got = ctx.sqa_solve(prob, prm)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got.replica_energies, want.replica_energies)
    np.testing.assert_array_equal(got.best_spins, want.best_spins)


def test_nmfa_gives_up():
    prob = sb.Problem.from_dense(instances.complete_pm1(600, seed=1))
    prm = sb.NmfaParams.default(stages=10, samples=96, seed=2, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    try:
        want = ctx.nmfa_solve(prob, prm)
        _expires(ctx, lambda: ctx.nmfa_solve(prob, prm), 5)
        got = ctx.nmfa_solve(prob, prm)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got.samples, want.samples)
