"""The multi-step kernel (sb_run.cuh) at the edges of its tiles, rings and waves, bit for bit against the
CPU oracle or against the same solve by another path."""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances
from oracle import binding as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sb.Context(0)
    yield c
    c.close()


def _check(res, J, h, R, steps, seed, c0):
    x, y = orc.init_uniform(J.shape[0], R, seed)
    orc.sb_run_f32(2, J, h, x, y, steps, 1.0, c0, 1.25)
    np.testing.assert_array_equal(res.final_x, x)
    np.testing.assert_array_equal(res.final_y, y)
    np.testing.assert_array_equal(res.replica_energies, orc.energies_of_x(J, h, x))


@pytest.mark.parametrize("n,R", [
    (1, 32), (31, 33), (128, 64), (129, 32),  # one and two spin tiles; one chunk (a stage's second half empty)
    (257, 65),                                # two chunks, the second's words mostly past the spins
    (600, 500),                               # three chunks: an odd tail; 32-replica items
    (1111, 700),                              # 64-replica items, one per CTA
    (2000, 600),                              # two 64-replica items per CTA, the last CTAs' second one missing
    (2300, 96),                               # nine chunks, the most that stay resident
])
def test_single_instance(ctx, n, R):
    J = instances.erdos_renyi(n, 0.4, seed=n, jmax=4, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-2, 3, n).astype(np.float32)
    prob = sb.Problem.from_dense(J, h)
    steps = 8 if n > 1000 else 20
    prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=5, field_mode=sb.FIELD_TC)
    res = ctx.solve(prob, prm, want_state=True)
    assert res.field_dtype == "fp4e2m1"
    _check(res, J, h, R, steps, 5, prob.default_c0())


@pytest.mark.parametrize("count,n,R,jmax", [
    (160, 130, 64, 1),   # E2M1: 320 items of two tiles, more than two per CTA hold: two waves
    (160, 130, 32, 9),   # E2M3: up to six 32-replica items per CTA, three here, streamed J
    (3, 1300, 64, 12),   # E2M3 rows too long to stay resident (11 chunks)
    (3, 1100, 100, 12),  # resident E2M3 rows, two replica tiles
    (2, 2600, 40, 3),    # E2M1 rows too long to stay resident (11 chunks), an odd chunk count
])
def test_batches(ctx, count, n, R, jmax):
    Js = [instances.erdos_renyi(n - (k % 3), 0.5, seed=100 + k, jmax=jmax, allow_zero=True) for k in range(count)]
    for J in Js:
        J[0, 1] = J[1, 0] = jmax  # the operand type the case is about
    probs = [sb.Problem.from_dense(J) for J in Js]
    steps = 7
    prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=40, field_mode=sb.FIELD_TC)
    batch = ctx.batch(probs, prm, want_state=True)
    res = batch.run()
    for k in range(0, count, max(1, count // 12)):
        _check(res[k], Js[k], None, R, steps, 40 + k, probs[k].default_c0())
    again = batch.run()
    for a, b in zip(res, again):
        np.testing.assert_array_equal(a.final_x, b.final_x)
        np.testing.assert_array_equal(a.replica_energies, b.replica_energies)
    batch.close()


def test_instance_beyond_a_wave(ctx):
    """4096 replicas of 700 spins are more items than a wave holds: that instance takes one launch per step
    beside one that runs in a wave."""
    Js = [instances.erdos_renyi(n, 0.5, seed=n, jmax=2, allow_zero=True) for n in (700, 200)]
    probs = [sb.Problem.from_dense(J) for J in Js]
    prm = sb.Params.default(sb.DSB, steps=6, replicas=4096, seed=3, field_mode=sb.FIELD_TC)
    batch = ctx.batch(probs, prm, want_state=True)
    res = batch.run()
    for k, J in enumerate(Js):
        x, y = orc.init_uniform(J.shape[0], 4096, 3 + k)
        orc.sb_run_f32(2, J, None, x, y, 6, 1.0, probs[k].default_c0(), 1.25)
        np.testing.assert_array_equal(res[k].final_x, x)
        np.testing.assert_array_equal(res[k].final_y, y)
    batch.close()


def test_trace_and_untraced_solves_agree(ctx):
    """A traced solve runs the kernel that exchanges operands, an untraced one the tagged words."""
    J = instances.complete_pm1(900, seed=4)
    prob = sb.Problem.from_dense(J)
    out = [ctx.solve(prob, sb.Params.default(sb.DSB, steps=300, replicas=256, seed=9, trace=t), want_state=True)
           for t in (0, 1)]
    np.testing.assert_array_equal(out[0].final_x, out[1].final_x)
    np.testing.assert_array_equal(out[0].final_y, out[1].final_y)
    np.testing.assert_array_equal(out[0].replica_energies, out[1].replica_energies)
