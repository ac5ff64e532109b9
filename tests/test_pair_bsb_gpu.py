"""The CTA-pair form of bSB on split operands (BF16 hi + lo by default, FP16 on request) against the single-CTA form
(SB_TC_PAIR=0), bit for bit: both add the same products into the same FP32 segments in the same order.

Sizes sit on the edges of the pair's 256 rows, the 64-spin chunks and their segments, and the replica tiles.
"""
import time

import numpy as np
import pytest

import annealing_gb300 as sb

pytestmark = pytest.mark.gpu

SB_ERR_TIMEOUT = 7


def _problem(n, fields):
    rng = np.random.default_rng(n)
    J = rng.normal(size=(n, n)).astype(np.float32) / np.float32(np.sqrt(n))
    J = np.triu(J, 1)
    h = rng.normal(size=n).astype(np.float32) if fields else None
    return sb.Problem.from_dense((J + J.T).astype(np.float32), h)


def _solve(prob, R, steps, dtype, pair, monkeypatch):
    if pair is None:
        monkeypatch.delenv("SB_TC_PAIR", raising=False)
    else:
        monkeypatch.setenv("SB_TC_PAIR", pair)
    ctx = sb.Context(0)
    try:
        prm = sb.Params.default(sb.BSB, steps=steps, replicas=R, seed=5, field_mode=sb.FIELD_TC, operand_dtype=dtype)
        return ctx.solve(prob, prm, want_state=True)
    finally:
        ctx.close()


@pytest.mark.parametrize("n,R,steps,dtype,pair,fields", [
    (130, 65, 9, "bf16", "1", True),      # two tiles, the second of two rows; one segment
    (512, 128, 1, "bf16", "1", False),    # exactly one segment of eight chunks
    (513 + 127, 100, 7, "bf16", "0", True),  # five tiles: single CTAs either way
    (700, 100, 20, "bf16", None, True),   # six tiles, two segments, the second short
    (1000, 128, 20, "bf16", None, False),
    (1409, 129, 9, "bf16", None, True),   # twelve tiles, the last of one row; two replica tiles, the second of one
    (2048, 256, 8, "bf16", None, False),  # whole tiles and segments
    (256, 128, 12, "fp16", "1", True),    # FP16 hi + lo: segments of two chunks
    (1000, 200, 9, "fp16", "1", False),
])
def test_pair_equals_single(n, R, steps, dtype, pair, fields, monkeypatch):
    prob = _problem(n, fields)
    dt = sb.OPERAND_FP16X2 if dtype == "fp16" else sb.OPERAND_BF16X2
    a = _solve(prob, R, steps, dt, pair, monkeypatch)
    b = _solve(prob, R, steps, dt, "0", monkeypatch)
    np.testing.assert_array_equal(a.final_x, b.final_x)
    np.testing.assert_array_equal(a.final_y, b.final_y)
    np.testing.assert_array_equal(a.best_spins, b.best_spins)


def test_wait_expires_then_context_solves(monkeypatch):
    """One unit leaves out its published flag (injected on the host): the waits of both CTAs of every pair expire, the
    call returns its status and the context stays usable."""
    monkeypatch.delenv("SB_TC_PAIR", raising=False)
    prob = _problem(1000, False)
    prm = sb.Params.default(sb.BSB, steps=24, replicas=128, seed=5, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    try:
        want = ctx.solve(prob, prm, want_state=True)
        ctx.set_wait_limit(1_000_000)
        ctx.debug_skip_publish(12)
        t0 = time.perf_counter()
        with pytest.raises(sb.SBError) as ei:
            ctx.solve(prob, prm)
        assert ei.value.status == SB_ERR_TIMEOUT, str(ei.value)
        assert time.perf_counter() - t0 < 0.5
        ctx.set_wait_limit(0)
        got = ctx.solve(prob, prm, want_state=True)
        np.testing.assert_array_equal(got.final_x, want.final_x)
    finally:
        ctx.close()
