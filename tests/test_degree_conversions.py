"""The FP32 degree conversions of the plain form's target chain equal the
reference's double-precision ones, (double)a * M_PI / 180.0 and
(double)v / M_PI rounded to FP32 (FIPkernels.cu:96-97, 145), for every FP32 value
of a binade: both forms scale with powers of two, so that binade stands for all.
Exact comparison: the results are the same numbers or they are not."""
import math
import os
import re

import numpy as np
import pytest

HEADER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fastimagingpipe_b200",
                      "csrc", "fip_refmath.cuh")


def constant(name):
    with open(HEADER) as f:
        text = re.search(r"constexpr float %s = ([-0-9a-fx.p]+)f;" % name, f.read()).group(1)
    v = float.fromhex(text)
    assert float(np.float32(v)) == v
    return v


def fma32(a, b, c):
    """FP32 fma(a, b, c) of FP32 values held in FP64: the product is exact there,
    the sum is rounded to odd (so that rounding it to FP32 rounds only once)."""
    p = a * b
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    bits = s.view(np.int64)
    step = np.where((err > 0) == (s > 0), 1, -1)
    bits += np.where((err != 0) & (bits & 1 == 0), step, 0)
    return bits.view(np.float64).astype(np.float32)


@pytest.mark.parametrize("hi,lo,exact", [
    ("kDegToRadHi", "kDegToRadLo", lambda v: (v * math.pi) / 180.0),
    ("kRadToDeg180Hi", "kRadToDeg180Lo", lambda v: v / math.pi),
])
def test_every_mantissa(hi, lo, exact):
    h, l = constant(hi), constant(lo)
    for part in np.array_split(np.arange(0x42000000, 0x42800000, dtype=np.uint32), 8):
        v = part.view(np.float32).astype(np.float64)
        low = (v * l).astype(np.float32).astype(np.float64)
        got = fma32(v, np.float64(h), low)
        want = exact(v).astype(np.float32)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
