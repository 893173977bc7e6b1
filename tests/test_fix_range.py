"""Conversions of the fixed-point transforms (csrc/sb_fix.cuh) at the ends of
the range, on the host: FP32 blocks of subnormal numbers alone keep them."""
import numpy as np

from test_fix import lib  # noqa: F401


def test_blocks_of_fp32_subnormals(lib):  # noqa: F811
    for bits in (57, 59, 61):
        for x in (1e-40, -1e-42, 2.0 ** -149, 2.0 ** -127, 1.17549421e-38):
            xf = np.float32(x)
            assert lib.fix_roundf(xf, xf, bits) == xf
    assert lib.fix_roundf(0.0, 0.0, 57) == 0.0
