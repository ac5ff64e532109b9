"""The block form of fully-connected SQA (fields on the tensor cores, |J| <= 4, up to 64 slices, 128 spins or more)
against the CPU oracle, bit for bit: integers throughout, so no tolerance.

Sizes sit on the edges of the blocks of 64 iterations, the 128-row and 256-column tiles, the 32-slice warps and the
magnitude planes, on both sides of the dispatch rule.
"""
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


def _oracle(J, M, R, steps, rng, seed):
    s, rnd = orc.sqa_init(J.shape[0], M, R, rng, seed)
    tr = orc.sqa_run(J, s, steps, rng, rnd=rnd, seed=seed)
    return s, tr


def _couplings(n, kind):
    if kind == "pm1":
        return instances.complete_pm1(n, seed=n)
    if kind == "ferro4":  # every field reaches (n - 1) 4: the ends of the 16-bit range
        return (4.0 * (1 - np.eye(n))).astype(np.float32)
    return instances.erdos_renyi(n, 0.6, n, jmax=int(kind[2:]), allow_zero=True)


@pytest.mark.parametrize("mode", [sb.SQA_RNG_HASH, sb.SQA_RNG_REFERENCE])
@pytest.mark.parametrize("n,M,R,steps,kind", [
    (127, 8, 2, 3, "pm1"),        # below the rule: the row-wise form
    (128, 1, 2, 4, "pm1"),        # smallest instance; one slice (its own Trotter neighbour)
    (128, 64, 2, 3, "er4"),       # every row in the block's 127, three planes
    (129, 2, 2, 4, "er3"),        # both neighbours are the same slice
    (161, 31, 2, 3, "pm1"),       # iterations M + n - 1 = 191 = 3 blocks less one
    (161, 32, 2, 3, "er2"),       # 192: whole blocks; one full warp
    (161, 33, 2, 3, "pm1"),       # 193: a block of one iteration; a second warp of one slice
    (255, 63, 3, 3, "er3"),
    (256, 64, 2, 3, "pm1"),       # whole column chunk
    (257, 65, 1, 2, "pm1"),       # above the rule: more slices than a tile holds
    (300, 40, 5, 2, "er5"),       # above the rule: |J| = 5
    (520, 48, 2, 2, "er4"),
    # more replicas than SMs: two per thread block, the last one alone
    (128, 64, 153, 2, "er4"),
    (130, 1, 301, 2, "pm1"),
    (161, 32, 153, 2, "er3"),
    (161, 33, 154, 2, "pm1"),
])
def test_blocks_match_the_oracle(ctx, n, M, R, steps, kind, mode):
    _check(ctx, _couplings(n, kind), M, R, steps, mode)


def test_fields_at_the_ends_of_16_bits(ctx):
    _check(ctx, _couplings(8191, "ferro4"), 2, 1, 3, sb.SQA_RNG_HASH)


def _check(ctx, J, M, R, steps, mode):
    prm = sb.SqaParams.default(trotter=M, steps=steps, replicas=R, rng_mode=mode, seed=91, trace=1)
    res = ctx.sqa_solve(sb.Problem.from_dense(J), prm, want_spins=True)
    s, tr = _oracle(J, M, R, steps, 1 if mode == sb.SQA_RNG_HASH else 0, 91)
    np.testing.assert_array_equal(res.final_spins, s)
    np.testing.assert_array_equal(res.energy_trace, tr.astype(np.float64))
    np.testing.assert_array_equal(res.replica_energies, tr[:, -1].astype(np.float64))
    assert res.energy_check_ok


@pytest.mark.parametrize("R", [31, 32, 33, 65, 100])
def test_reference_states_of_many_replicas(ctx, R):
    """Reference mode starts replicas in up to 32 rows, each jumping ahead in the xorshift sequence."""
    _check(ctx, _couplings(150, "pm1"), 5, R, 2, sb.SQA_RNG_REFERENCE)
