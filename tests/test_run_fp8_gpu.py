"""Untraced FP8 dSB solves (integer |J| <= 16 beyond E2M1) with all steps in one launch and signs exchanged as tagged
words, against the plain FP32 kernel, bit for bit: the fields are exact integers in both.

Sizes sit on the edges of the 128-spin tiles and chunks, the nine resident chunks, the 32- and 64-replica tiles and two
items to a CTA.
"""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,steps,fields", [
    (1, 32, 3, True),
    (127, 33, 12, False),
    (129, 65, 11, True),
    (700, 300, 8, True),
    (1152, 64, 10, False),    # nine chunks: resident rows
    (1153, 64, 11, True),     # ten: streamed
    (1300, 500, 6, False),    # 64-replica tiles
    (1300, 1000, 5, True),    # two to a CTA, streamed
    (1000, 1210, 5, False),   # two to a CTA, resident, the last one alone
    (4096, 40, 3, False),
])
def test_one_launch_fp8_equals_plain(n, R, steps, fields, monkeypatch):
    J = instances.erdos_renyi(n, 0.5, seed=n + R, jmax=16, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-3, 4, n).astype(np.float32) if fields else None
    prob = sb.Problem.from_dense(J, h)
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    ctx = sb.Context(0)
    try:
        got = []
        for mode, dt in ((sb.FIELD_TC, sb.OPERAND_FP8), (sb.FIELD_FP32, sb.OPERAND_AUTO)):
            prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=13, field_mode=mode, operand_dtype=dt)
            got.append(ctx.solve(prob, prm, want_state=True))
    finally:
        ctx.close()
    a, b = got
    assert a.field_dtype == "fp8e4m3" and a.steps_per_launch == steps
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
    np.testing.assert_array_equal(a.replica_energies, b.replica_energies)
    assert a.energy_check_ok
