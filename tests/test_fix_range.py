"""Conversions of the fixed-point transforms (csrc/sb_fix.cuh) at the ends of
the range, on the host: FP32 blocks of subnormal numbers alone keep them, and
results of any size below the range come out right or, below the smallest
normal number, as zero."""
import math

import numpy as np

from test_fix import lib  # noqa: F401


def test_blocks_of_fp32_subnormals(lib):  # noqa: F811
    for bits in (57, 59, 61):
        for x in (1e-40, -1e-42, 2.0 ** -149, 2.0 ** -127, 1.17549421e-38):
            xf = np.float32(x)
            assert lib.fix_roundf(xf, xf, bits) == xf
    assert lib.fix_roundf(0.0, 0.0, 57) == 0.0


def test_small_results(lib):  # noqa: F811
    for v in (1, -3, 1 << 40, -(1 << 60), (1 << 62) + 1):
        for t in range(-1300, -880, 7):
            exact = math.ldexp(float(v), t)
            got = lib.fix_out(v, t)
            if abs(exact) >= 2.0 ** -1022:
                assert got == exact, (v, t)
            else:
                assert got == 0.0, (v, t)
        for t in (-4000, -8000, -100000):
            assert lib.fix_out(v, t) == 0.0
