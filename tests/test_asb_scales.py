"""The FP32 form of the aSB local sub-steps (csrc/sb_asb.cuh) far from the usual constants: a large Kerr constant or time
step multiplies what a product near the subnormals has lost, and the bits still have to be the double evaluation's."""
import numpy as np
import pytest

from oracle import binding as orc
from test_asb_local import _values, local  # noqa: F401


@pytest.mark.parametrize("kind", ["unit", "tiny", "special"])
@pytest.mark.parametrize("dt,detune,kerr", [(0.5, 1.0, 1e10), (0.5, 1.0, -1e30), (1e6, 1.0, 1.0), (-1e20, 1.0, 1.0),
                                            (1e12, 1e-12, 1.0), (0.5, 1e-30, 1e3), (1e-30, 1e30, 1e30)])
def test_bits_of_the_double_evaluation(local, kind, dt, detune, kerr):  # noqa: F811
    rng = np.random.default_rng(len(kind))
    for amp in (0.0, 0.525, 1.0):
        with np.errstate(all="ignore"):
            x, y = (v.astype(np.float32) for v in _values(kind, rng, 200000))
        wx, wy = x.copy(), y.copy()
        orc.asb_local(wx, wy, amp, 1, dt, detune, kerr)
        local(x.size, x.ctypes.data, y.ctypes.data, amp, 1, dt, detune, kerr)
        for a, w in ((x, wx), (y, wy)):
            np.testing.assert_array_equal(np.isnan(a), np.isnan(w))
            f = ~np.isnan(w)
            np.testing.assert_array_equal(a.view(np.uint32)[f], w.view(np.uint32)[f])
