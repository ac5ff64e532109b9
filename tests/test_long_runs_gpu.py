"""Anneals longer than a step's tag or a launch: the 16-bit tags of the sign exchange through L2 wrap, and a wave's steps
are split over launches of 2^20."""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


def test_sign_tags_wrap(monkeypatch):
    """|J| <= 3 beyond 1024 spins: one launch with its signs exchanged through L2, against a launch per step."""
    prob = sb.Problem.from_dense(instances.erdos_renyi(1025, 0.5, seed=2, jmax=3, allow_zero=True))
    prm = sb.Params.default(sb.DSB, steps=65536 + 40, replicas=1, seed=5, field_mode=sb.FIELD_FP32)
    out = []
    for env in (None, "0"):
        monkeypatch.delenv("SB_PLAIN_PERSIST", raising=False) if env is None else monkeypatch.setenv("SB_PLAIN_PERSIST", env)
        ctx = sb.Context(0)
        try:
            out.append(ctx.solve(prob, prm, want_state=True))
        finally:
            ctx.close()
    assert [r.steps_per_launch for r in out] == [prm.steps, 1]
    np.testing.assert_array_equal(out[0].final_x, out[1].final_x)
    np.testing.assert_array_equal(out[0].final_y, out[1].final_y)


def test_a_wave_takes_several_launches():
    """Against the same anneal on bit planes, in one launch."""
    prob = sb.Problem.from_dense(instances.complete_pm1(40, seed=1))
    steps = (1 << 20) + 3
    ctx = sb.Context(0)
    batch = None
    try:
        batch = ctx.batch([prob], sb.Params.default(sb.DSB, steps=steps, replicas=2, seed=5, field_mode=sb.FIELD_TC),
                          want_state=True)
        a = batch.run()[0]
        b = ctx.solve(prob, sb.Params.default(sb.DSB, steps=steps, replicas=2, seed=5, field_mode=sb.FIELD_FP32), want_state=True)
    finally:
        if batch:
            batch.close()
        ctx.close()
    assert a.steps_per_launch == 1 << 20 and b.steps_per_launch == steps
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
