"""Untraced BF16 dSB solves (integer |J| <= 256) with all steps in one launch, the couplings as 16 hi + lo in E4M3 and the
signs exchanged as tagged words, against the plain FP32 kernel, bit for bit: the fields are exact integers in both.

Sizes sit on the edges of the 128-spin tiles and chunks, the four resident pairs of chunks, the 32- and 64-replica tiles
and two items to a CTA. Couplings cover -256 .. 256; the last cases have all spins aligned by couplings of 255, whose
fields are the largest odd multiples.
"""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,steps,fields,aligned", [
    (1, 32, 3, True, False),
    (127, 33, 12, False, False),
    (129, 65, 11, True, False),
    (512, 64, 10, False, False),   # four pairs of chunks: resident rows
    (513, 300, 11, True, False),   # five: streamed
    (500, 2400, 6, True, False),   # two 64-replica items to a CTA, resident, the last one alone
    (1300, 500, 6, False, False),  # 64-replica tiles
    (1300, 1000, 5, True, False),  # two to a CTA, streamed
    (640, 700, 30, True, True),
    (4096, 40, 20, False, True),
])
def test_one_launch_bf16_equals_plain(n, R, steps, fields, aligned, monkeypatch):
    if aligned:
        J = np.full((n, n), 255, np.float32)
        np.fill_diagonal(J, 0)
    else:
        J = instances.erdos_renyi(n, 0.5, seed=n + R, jmax=256, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-3, 4, n).astype(np.float32) if fields else None
    prob = sb.Problem.from_dense(J, h)
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    ctx = sb.Context(0)
    try:
        got = []
        for mode, dt in ((sb.FIELD_TC, sb.OPERAND_BF16), (sb.FIELD_FP32, sb.OPERAND_AUTO)):
            prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=13, field_mode=mode, operand_dtype=dt)
            got.append(ctx.solve(prob, prm, want_state=True))
    finally:
        ctx.close()
    a, b = got
    assert a.field_dtype == "bf16" and a.steps_per_launch == steps
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
    np.testing.assert_array_equal(a.replica_energies, b.replica_energies)
    assert a.energy_check_ok
