"""Plain FP32 dSB with integer couplings up to 127 in one launch (bit planes and popcounts; one CTA up to 512 spins, a
cluster above) against the general one-launch-per-step kernel, bit for bit: the fields are exact integers in both.

Sizes sit on the edges of words, register forms, the one-CTA limit and the clusters (up to sixteen CTAs), and on both
sides of the dispatch rule.
"""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


def _solve(prob, n, R, steps, seed, persist, monkeypatch):
    if persist:
        monkeypatch.delenv("SB_PLAIN_PERSIST", raising=False)
    else:
        monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    ctx = sb.Context(0)
    try:
        prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=seed, field_mode=sb.FIELD_FP32)
        return ctx.solve(prob, prm, want_state=True)
    finally:
        ctx.close()


@pytest.mark.parametrize("n,jmax,R,steps,fields", [
    (1, 1, 1, 3, True),
    (31, 1, 2, 1, False),
    (33, 7, 3, 2, True),
    (128, 1, 1, 100, False),
    (129, 3, 2, 40, True),
    (256, 7, 5, 40, False),
    (257, 1, 9, 41, True),
    (511, 3, 2, 60, False),
    (512, 7, 12, 30, True),
    (513, 1, 1, 2, False),     # a cluster of five CTAs, the last with one row
    (640, 3, 3, 60, True),
    (1000, 7, 2, 61, False),   # eight
    (1024, 3, 40, 20, True),
    (1025, 1, 1, 1, True),     # nine
    (1111, 1, 12, 60, False),
    (1900, 1, 3, 40, True),    # fifteen
    (2048, 1, 2, 100, False),  # sixteen
    (1025, 3, 1, 30, False),   # more planes than registers hold: signs through L2
    (300, 8, 2, 30, True),     # four planes
    (64, 127, 3, 40, True),    # seven, one CTA
    (256, 31, 5, 40, False),
    (511, 64, 2, 40, True),    # seven, a cluster of four
    (1024, 15, 2, 40, False),  # four, eight CTAs
    (1000, 16, 1, 20, True),   # five planes of this size: signs through L2
    (300, 128, 2, 30, False),  # |J| above 127
    (2049, 1, 1, 20, False),
])
def test_sign_solve_equals_per_step(n, jmax, R, steps, fields, monkeypatch):
    J = instances.erdos_renyi(n, 0.7, seed=n + jmax, jmax=jmax, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-3, 4, n).astype(np.float32) if fields else None
    prob = sb.Problem.from_dense(J, h)
    a = _solve(prob, n, R, steps, 11, True, monkeypatch)
    b = _solve(prob, n, R, steps, 11, False, monkeypatch)
    assert b.steps_per_launch == 1
    if n <= 512 and jmax <= 127 or n <= 1024 and jmax <= 15 or n <= 2048 and jmax == 1:
        assert a.steps_per_launch == steps and a.kernel_launches == 3
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
    np.testing.assert_array_equal(a.replica_energies, b.replica_energies)
    np.testing.assert_array_equal(a.best_spins, b.best_spins)


def test_a_cached_plan_takes_other_couplings(monkeypatch):
    """One context, one shape: small integers, then real couplings, then integers again."""
    n = 300
    rng = np.random.default_rng(3)
    real = rng.normal(size=(n, n)).astype(np.float32)
    real = np.triu(real, 1) + np.triu(real, 1).T
    problems = [sb.Problem.from_dense(J) for J in (instances.complete_pm1(n, seed=1), real,
                                                   instances.erdos_renyi(n, 0.5, 2, jmax=5, allow_zero=True))]
    monkeypatch.delenv("SB_PLAIN_PERSIST", raising=False)
    ctx = sb.Context(0)
    try:
        prm = sb.Params.default(sb.DSB, steps=50, replicas=2, seed=4, field_mode=sb.FIELD_FP32, c0=0.05)
        got = [ctx.solve(p, prm, want_state=True) for p in problems]
    finally:
        ctx.close()
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    for p, a in zip(problems, got):
        ctx = sb.Context(0)
        try:
            b = ctx.solve(p, prm, want_state=True)
        finally:
            ctx.close()
        np.testing.assert_array_equal(a.final_x, b.final_x)
        np.testing.assert_array_equal(a.final_y, b.final_y)


@pytest.mark.parametrize("n,jmax,R,planes", [
    (100, 1, 64, True),
    (256, 4, 300, True),     # three planes, one CTA
    (512, 1, 512, True),     # 134e6: the one-CTA limit
    (512, 1, 514, False),
    (513, 3, 100, True),     # 53e6, a cluster of five
    (513, 3, 130, False),    # 68e6
    (640, 7, 65, True),      # FP8 on the tensor cores: 205e6, 640 counting as 1024
    (640, 7, 66, False),
    (88, 16, 599, True),
    (200, 100, 40, True),    # BF16 on the tensor cores
    (200, 200, 40, False),   # more planes than the kernel has
])
def test_automatic_mode_takes_the_faster_form(n, jmax, R, planes):
    J = instances.erdos_renyi(n, 0.7, seed=n + R, jmax=jmax, allow_zero=True)
    J[0, 1] = J[1, 0] = jmax
    prob = sb.Problem.from_dense(J)
    ctx = sb.Context(0)
    try:
        auto = ctx.solve(prob, sb.Params.default(sb.DSB, steps=25, replicas=R, seed=3), want_state=True)
        tc = ctx.solve(prob, sb.Params.default(sb.DSB, steps=25, replicas=R, seed=3, field_mode=sb.FIELD_TC), want_state=True)
    finally:
        ctx.close()
    assert auto.field_mode == (sb.FIELD_FP32 if planes else sb.FIELD_TC) and tc.field_mode == sb.FIELD_TC
    np.testing.assert_array_equal(auto.final_x, tc.final_x)
    np.testing.assert_array_equal(auto.final_y, tc.final_y)
    np.testing.assert_array_equal(auto.replica_energies, tc.replica_energies)
    assert auto.energy_check_ok
