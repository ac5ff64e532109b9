"""The states may go to any memory that a copy from the device reaches: an array in device or pinned memory, large enough
that the library would make a pageable one's pages present beforehand, gets what a pageable one gets."""
import ctypes as C

import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances
from annealing_gb300.sb import _ResultBuffers, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, R = 700, 128  # 358 KB of states


@pytest.mark.parametrize("where", ["cuda", "pinned"])
def test_states_to_other_memory(where):
    if where == "cuda":
        x, y = (torch.zeros((R, N), device="cuda") for _ in range(2))
    else:
        x, y = (torch.zeros((R, N), pin_memory=True) for _ in range(2))
    torch.cuda.synchronize()
    prob = sb.Problem.from_dense(instances.complete_pm1(N, seed=1))
    prm = sb.Params.default(sb.DSB, steps=20, replicas=R, seed=3, field_mode=sb.FIELD_TC)
    ctx = sb.Context(0)
    plan, batch = ctx.plan(prob, prm, want_state=True), ctx.batch([prob], prm, want_state=True)
    try:
        for run, h, want in ((lib().sb_plan_run, plan.h, plan.run(seed=3)), (lib().sb_batch_run, batch.h, batch.run(seed=3)[0])):
            buf = _ResultBuffers(N, prm, True)
            buf.r.final_x = C.cast(C.c_void_p(x.data_ptr()), type(buf.r.final_x))
            buf.r.final_y = C.cast(C.c_void_p(y.data_ptr()), type(buf.r.final_y))
            x.zero_()
            y.zero_()
            torch.cuda.synchronize()
            assert run(h, 3, C.byref(buf.r)) == 0
            np.testing.assert_array_equal(x.cpu().numpy(), want.final_x)
            np.testing.assert_array_equal(y.cpu().numpy(), want.final_y)
    finally:
        batch.close()
        plan.close()
        ctx.close()
