"""Energies of the register tiles (32 rows x 16 replicas a CTA), summed by shuffles and over four warps: at the edges of a
tile's rows, of its two halves of eight replicas and of a warp's eight rows, against the CPU oracle. Integer couplings and
fields exactly; real ones, whose fields are the oracle's FP32 sums, to the order of some n additions in double."""
import numpy as np
import pytest

import annealing_gb300 as sb
from annealing_gb300 import instances
from oracle import binding as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(1, 8), (7, 9), (8, 16), (9, 17), (31, 24), (32, 25), (33, 40), (63, 33), (65, 15),
                                 (700, 23), (3001, 5)])
@pytest.mark.parametrize("variant", [sb.ASB, sb.BSB, sb.DSB])
def test_traced_integers(n, R, variant, monkeypatch):
    monkeypatch.setenv("SB_PLAIN_PERSIST", "0")
    J = instances.erdos_renyi(n, 0.6, seed=n, jmax=5, allow_zero=True) if n > 1 else np.zeros((1, 1), np.float32)
    h = np.random.default_rng(n).integers(-4, 5, n).astype(np.float32) if variant != sb.ASB else None
    steps = 6
    ctx = sb.Context(0)
    try:
        res = ctx.solve(sb.Problem.from_dense(J, h), sb.Params.default(variant, steps=steps, replicas=R, seed=2, trace=1, trace_all=1,
                                                                       field_mode=sb.FIELD_FP32), want_state=True)
    finally:
        ctx.close()
    np.testing.assert_array_equal(res.replica_energies, orc.energies_of_x(J, h, res.final_x))
    np.testing.assert_array_equal(res.energy_trace_all[-1], res.replica_energies)
    if variant != sb.ASB:
        x, _ = orc.init_uniform(n, R, 2)
        np.testing.assert_array_equal(res.energy_trace_all[0], orc.energies_of_x(J, h, x))


@pytest.mark.parametrize("n,R", [(40, 9), (700, 40)])
def test_real_couplings(n, R):
    """More replicas than are refined in FP64: the others keep the tile's energies, FP32 fields summed in double
    (n 2^-24 of the terms' sum of magnitudes, at most)."""
    J = instances.gaussian(n, seed=n)[0]
    ctx = sb.Context(0)
    try:
        res = ctx.solve(sb.Problem.from_dense(J), sb.Params.default(sb.BSB, steps=20, replicas=R, seed=2, field_mode=sb.FIELD_FP32),
                        want_state=True)
    finally:
        ctx.close()
    s = np.where(res.final_x > 0, 1.0, -1.0)
    exact = -0.5 * np.einsum("ri,ij,rj->r", s, J.astype(np.float64), s)
    np.testing.assert_allclose(res.replica_energies, exact, rtol=0, atol=n * 2.0**-24 * np.abs(J).sum() / 2)
    assert res.energy_check_ok
