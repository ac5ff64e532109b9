"""Wait limits shorter than a copy takes count as the least one: solves under a limit of one clock give what they give
under the default, on every tensor-core kernel that runs a solve."""
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
