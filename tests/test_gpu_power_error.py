"""Rounding of the powers (F^2)^q of half-integer q, from registers: no larger than that of
pow(F^2, q).  psi = (a, 0) with a 26-bit a has F = a^2 exactly for I and Z and 0 for X and Y, so
that the sum is twice one power."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A = np.random.default_rng(42).integers(1 << 25, 1 << 26, size=4000) / float(1 << 26)


def rms(value, q):
    exact = (A.astype(np.longdouble) ** 2) ** np.longdouble(2 * q)
    return float(np.sqrt(np.mean(((value.astype(np.longdouble) - exact) / exact) ** 2)))


@pytest.mark.parametrize("q", [1.5, 2.5, 3.5, 5.5, 6.5, 7.5, 8.5, 10.5, 11.5, 12.5, 13.5, 14.5, 15.5])
def test_no_larger_than_pow(ctx, hm, q):
    got = np.empty_like(A)
    for i, a in enumerate(A):
        _, m = ctx.sre_range(np.array([a, 0.0], dtype=complex), 0, 2, (q,), hm.HM_FP64)
        got[i] = m.sum() / 2
    # 4000 values: the two rms are known to about 1 %; squaring F^2 instead of F is 3 to 5 % above
    assert rms(got, q) <= 1.02 * rms(np.power((A * A) ** 2, q), q)
