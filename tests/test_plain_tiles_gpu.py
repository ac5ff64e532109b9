"""The register-tile form of the plain FP32 field (32 rows x 16 replicas per CTA, 128 floats of K per
stage) at the edges of its tiles and ring, bit for bit against the CPU oracle."""
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


@pytest.mark.parametrize("n,R", [(1, 8), (3, 16), (31, 8), (32, 17), (33, 15), (128, 16), (129, 9), (511, 33),
                                 (641, 31), (1030, 24), (3001, 4)])
def test_dsb_tiles_bit_exact(ctx, n, R, monkeypatch):
    """Integer J with fields: the trajectory, the final energies and the per-step energies."""
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    J = instances.erdos_renyi(n, 0.5, seed=n, jmax=3, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-2, 3, n).astype(np.float32)
    steps = 12 if n < 2000 else 3
    prob = sb.Problem.from_dense(J, h)
    x, y = orc.init_uniform(n, R, 5)
    tr = orc.sb_run_f32(2, J, h, x, y, steps, 1.0, prob.default_c0(), 1.25, trace=True, trace_all=True)
    for trace in (0, 1):
        prm = sb.Params.default(sb.DSB, steps=steps, replicas=R, seed=5, field_mode=sb.FIELD_FP32, trace=trace,
                                trace_all=trace)
        res = ctx.solve(prob, prm, want_state=True)
        np.testing.assert_array_equal(res.final_x, x)
        np.testing.assert_array_equal(res.final_y, y)
        np.testing.assert_array_equal(res.replica_energies, orc.energies_of_x(J, h, x))
    np.testing.assert_array_equal(res.energy_trace_all, tr[1])


@pytest.mark.parametrize("n,R,stages", [(32, 8, 4), (130, 17, 3), (515, 16, 3), (1029, 25, 2)])
def test_nmfa_tiles_bit_exact(ctx, n, R, stages, monkeypatch):
    """Real-valued states: the oracle sums in the kernel's order, so a changed order shows."""
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    J = instances.nmfa_fully(n, seed=n)
    betas = sb.nmfa_schedule(100)[:stages]
    p = sb.NmfaParams.default(samples=R, seed=n, field_mode=sb.FIELD_FP32)
    res = ctx.nmfa_solve(sb.Problem.from_dense(J), p, betas=betas, want_states=True)
    st, sp, _ = orc.nmfa_run(J, R, betas, 0.15, 0.15, n)
    np.testing.assert_array_equal(res.states.view(np.uint32), st.view(np.uint32))
    np.testing.assert_array_equal(res.samples, sp)


def test_same_bits_alone_and_together(ctx):
    """A replica's aSB trajectory does not depend on how many run beside it: four replicas (one
    row per warp) equal the first four of twenty (tiles), from the reference's start values."""
    J = instances.complete_pm1(700, seed=3)
    prob = sb.Problem.from_dense(J)
    out = []
    for R in (4, 20):
        prm = sb.Params.default(sb.ASB, steps=20, replicas=R, init_mode=sb.INIT_REFERENCE)
        out.append(ctx.solve(prob, prm, want_state=True))
    np.testing.assert_array_equal(out[0].final_x.view(np.uint32), out[1].final_x[:4].view(np.uint32))
    np.testing.assert_array_equal(out[0].final_y.view(np.uint32), out[1].final_y[:4].view(np.uint32))
