"""The short f32 root and quotient and the f64 reciprocal against the device's
IEEE operations over the ranges they are used in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT, QUOTIENT, RECIPROCAL = 0, 1, 2


def _differ(ctx, which, first, count):
    out = np.zeros(2, dtype=np.uint64)
    ctx.check(ctx.lib.ldsc_debug_approx(ctx.h, which, first, count, out.ctypes.data))
    print("differ %d of %d, at most %d places" % (out[0], count, out[1]))
    return int(out[0]), int(out[1])


def test_every_root_of_the_range_is_the_ieee_root(ctx):
    lo, hi = np.float32([8.0, 2.0 ** 30]).view(np.uint32)
    assert _differ(ctx, ROOT, int(lo), int(hi) - int(lo)) == (0, 0)


def test_quotients_are_within_a_place(ctx):
    """The remainder is exact and the first quotient within two places, so the
    corrected one is the neighbour at worst, and only on a near tie."""
    count = 3 * 10 ** 9
    differ, places = _differ(ctx, QUOTIENT, 0, count)
    assert places <= 1 and differ <= count * 1e-6


def test_reciprocals_are_within_a_place(ctx):
    """e^3 < 2^-57 of the value and two roundings: the neighbour at worst."""
    count = 3 * 10 ** 9
    differ, places = _differ(ctx, RECIPROCAL, 0, count)
    assert places <= 1 and differ <= count // 2
