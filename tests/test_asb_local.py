"""The FP32 form of the aSB local sub-steps (csrc/sb_asb.cuh, compiled here as host code) gives the
bits of the double evaluation: the reference's operations in the oracle (oracle_asb_local)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import binding as orc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def local(tmp_path_factory):
    d = tmp_path_factory.mktemp("asb")
    src, so = d / "asb.cpp", d / "asb.so"
    src.write_text('#include <cmath>\nusing std::isfinite;\nusing std::signbit;\n'
                   '#include "%s"\n' % os.path.join(ROOT, "annealing_gb300", "csrc", "sb_asb.cuh") +
                   'extern "C" void run(long n, float *x, float *y, float a, int m, float h, float d, float k) {\n'
                   '  for (long i = 0; i < n; ++i) sbasb::local(x[i], y[i], a, m, h, d, k);\n}\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC", str(src),
                    "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).run
    fn.argtypes = [C.c_long, C.c_void_p, C.c_void_p, C.c_float, C.c_int, C.c_float, C.c_float, C.c_float]
    return fn


def _values(kind, rng, n):
    u = lambda: rng.uniform(-1, 1, n)  # noqa: E731
    if kind == "unit":
        return u(), u()
    if kind == "grid":  # few bits: sums that lie on rounding boundaries
        return np.rint(u() * 4096) / 4096, np.rint(u() * 65536) / 65536
    if kind == "halfway":  # y half an ulp of the result away from the other term
        x = np.rint(u() * 256) / 256
        return x, np.ldexp(np.rint(u() * 3), -rng.integers(20, 60, n))
    if kind == "tiny":
        return np.ldexp(u(), -rng.integers(0, 160, n)), np.ldexp(u(), -rng.integers(0, 160, n))
    if kind == "huge":
        return np.ldexp(u(), rng.integers(0, 128, n)), np.ldexp(u(), rng.integers(0, 128, n))
    x, y = u(), u()  # special values
    sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 3e38])
    return np.where(rng.random(n) < 0.5, sp[rng.integers(0, 8, n)], x), np.where(rng.random(n) < 0.5, sp[rng.integers(0, 8, n)], y)


@pytest.mark.parametrize("kind", ["unit", "grid", "halfway", "tiny", "huge", "special"])
@pytest.mark.parametrize("m,dt,detune,kerr", [(2, 0.5, 1.0, 1.0), (1, 0.3, 0.7, 2.1), (3, -0.25, -1.0, 0.0)])
def test_bits_of_the_double_evaluation(local, kind, m, dt, detune, kerr):
    rng = np.random.default_rng(len(kind) + 10 * m)
    for amp in (0.0, 0.35, 0.99, 1.0):
        with np.errstate(all="ignore"):
            x, y = (v.astype(np.float32) for v in _values(kind, rng, 100000))
        wx, wy = x.copy(), y.copy()
        orc.asb_local(wx, wy, amp, m, dt, detune, kerr)
        local(x.size, x.ctypes.data, y.ctypes.data, amp, m, dt, detune, kerr)
        np.testing.assert_array_equal(np.isnan(x), np.isnan(wx))
        np.testing.assert_array_equal(np.isnan(y), np.isnan(wy))
        f, g = ~np.isnan(wx), ~np.isnan(wy)
        np.testing.assert_array_equal(x.view(np.uint32)[f], wx.view(np.uint32)[f])
        np.testing.assert_array_equal(y.view(np.uint32)[g], wy.view(np.uint32)[g])
