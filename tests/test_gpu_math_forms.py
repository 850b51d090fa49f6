"""The step's own square root, reciprocal products and Box-Muller forms over
their whole input ranges on the device (tests/native/math_check.cu): the same
bits as sqrtf, the step's division and the general Box-Muller."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flexpart-gpu_b200", "lib",
                   "libfpg_check.so")
CHECKS = ["square root", "quotient", "radius", "radius, packed lane 0", "radius, packed lane 1", "angle",
          "angle, packed lane 0", "angle, packed lane 1"]


@pytest.mark.parametrize("unit", ["step", "plain"])
def test_every_input_gives_the_same_bits(unit):
    """`unit`: the flags of the step's units, and of the others (which use the
    scalar Box-Muller form)."""
    out = np.zeros(2 * len(CHECKS) + 1, np.uint64)
    check = getattr(ctypes.CDLL(LIB), f"math_check_{unit}")
    assert check(ctypes.c_void_p(out.ctypes.data)) == 0
    assert out[-1] != 0                                     # a word whose radius is exactly 1 was found
    differ = {name: (int(out[2 * k]), int(out[2 * k + 1])) for k, name in enumerate(CHECKS) if out[2 * k]}
    assert not differ, f"inputs that differ, and the first of them: {differ}"
