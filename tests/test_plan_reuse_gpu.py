"""One context, one shape, one plan: problems of different kinds in turn give what each gives in a context of its own
(energies, best replica and spins, and the host re-check, besides the states)."""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


def _problem(kind, n):
    if kind == "real":
        A = np.triu(np.random.default_rng(3).normal(size=(n, n)).astype(np.float32), 1)
        return sb.Problem.from_dense(A + A.T)
    if kind == "large":  # integers that BF16 hi + lo (16 bits) does not hold; n |J| < 2^24
        J = instances.erdos_renyi(n, 0.7, seed=5, jmax=1, allow_zero=True)
        J = np.triu(J * np.random.default_rng(6).integers(35000, 35999, (n, n)).astype(np.float32) * 2 + np.sign(J), 1)
        return sb.Problem.from_dense((J + J.T).astype(np.float32))
    return sb.Problem.from_dense(instances.erdos_renyi(n, 0.7, seed=int(kind), jmax=int(kind), allow_zero=True))


@pytest.mark.parametrize("n,R,mode,dtype,kinds", [
    (300, 2, sb.FIELD_FP32, sb.OPERAND_AUTO, ("1", "real", "5")),
    (300, 20, sb.FIELD_FP32, sb.OPERAND_AUTO, ("1", "real", "5")),   # more replicas than are refined in FP64
    (300, 20, sb.FIELD_FP32, sb.OPERAND_AUTO, ("real", "3", "real")),
    (200, 40, sb.FIELD_TC, sb.OPERAND_BF16X2, ("real", "7", "large", "real")),
    (200, 40, sb.FIELD_TC, sb.OPERAND_BF16X2, ("7", "large")),
])
def test_energies_follow_the_problem(n, R, mode, dtype, kinds):
    prm = sb.Params.default(sb.DSB, steps=50, replicas=R, seed=4, field_mode=mode, operand_dtype=dtype, c0=0.05)
    problems = [_problem(k, n) for k in kinds]
    ctx = sb.Context(0)
    try:
        got = [ctx.solve(p, prm, want_state=True) for p in problems]
    finally:
        ctx.close()
    for kind, p, a in zip(kinds, problems, got):
        ctx = sb.Context(0)
        try:
            b = ctx.solve(p, prm, want_state=True)
        finally:
            ctx.close()
        np.testing.assert_array_equal(a.final_x, b.final_x)
        if kind == "real":  # blocks add their FP64 sums of some 10^5 terms in any order: 10^5 x 2^-53 of them
            np.testing.assert_allclose(a.replica_energies, b.replica_energies, rtol=1e-11)
        else:
            np.testing.assert_array_equal(a.replica_energies, b.replica_energies)
        np.testing.assert_array_equal(a.best_spins, b.best_spins)
        assert a.best_replica == b.best_replica
        assert a.energy_check_ok and b.energy_check_ok


def test_the_form_follows_the_problem():
    """Twelve replicas of 1000 spins fit no co-resident grid: integers take the one-launch bit planes whichever
    couplings the plan began with, real ones a launch per step."""
    n, R, steps = 1000, 12, 30
    prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=4, field_mode=sb.FIELD_FP32, c0=0.03)
    kinds = ("real", "1", "7", "real", "1")
    problems = {k: _problem(k, n) for k in kinds}
    ctx = sb.Context(0)
    try:
        got = [ctx.solve(problems[k], prm, want_state=True) for k in kinds]
    finally:
        ctx.close()
    for k, a in zip(kinds, got):
        ctx = sb.Context(0)
        try:
            b = ctx.solve(problems[k], prm, want_state=True)
        finally:
            ctx.close()
        assert a.steps_per_launch == b.steps_per_launch == (1 if k == "real" else steps)
        np.testing.assert_array_equal(a.final_x, b.final_x)
        np.testing.assert_array_equal(a.final_y, b.final_y)
