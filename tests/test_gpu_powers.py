"""Renyi indices outside {2, 3}: integers and half-integers from registers (powers and |F|),
every other index, or a list with one, through pow(); and the register splits of the sizes
that one warp holds.  Reference: the transforms in numpy."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu

QS = [(4.0,), (2.5,), (1.0, 1.5, 15.5, 16.0), (2.7,), (4.0, 2.7, 2.5), (16.0, 1.0)]


def _sums(psi, kb, ke, qs):
    dim, out = psi.size, np.zeros(len(qs))
    for k in range(kb, ke):
        b = psi[np.arange(dim) ^ (k ^ (k >> 1))]
        g = psi.real * (b.real + b.imag) + psi.imag * (b.imag - b.real)
        h = 1
        while h < dim:
            g = g.reshape(-1, 2, h)
            g = np.concatenate([g[:, :1] + g[:, 1:], g[:, :1] - g[:, 1:]], axis=1).reshape(-1)
            h *= 2
        out += [np.sum((g * g) ** q) for q in qs]
    return out


@pytest.mark.parametrize("qs", QS, ids=str)
@pytest.mark.parametrize("n", [1, 4, 7, 11, 12, 14, 15, 17, 20])
def test_range_powers(ctx, hm, n, qs):
    psi, full = rand_state(1 << n, 300 + n), 1 << n
    kb, ke = (0, min(full, 40)) if n <= 12 else (full // 2 - 1, full // 2 + 3)
    _, m = ctx.sre_range(psi, kb, ke, qs, hm.HM_FP64)
    # positive terms; F to n rounding steps of the largest values, q = 16 the 32nd power of it
    assert m.sum(axis=1) == pytest.approx(_sums(psi, kb, ke, qs), rel=1e-11)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("qs", [(2.0,), (3.0, 2.0), (4.0,), (2.7,)], ids=str)
@pytest.mark.parametrize("n", range(1, 12))
def test_one_warp_sizes(ctx, hm, n, qs, precision):
    psi, full = rand_state(1 << n, 400 + n), 1 << n
    # a full sweep, ranges that leave a warp's group of X-strings part empty, the last one alone
    for kb, ke in {(0, full), (0, 1), (1, min(full, 4)), (full // 3, full // 2 + 1), (full - 1, full)}:
        _, m = ctx.sre_range(psi, kb, ke, qs, hm.PRECISIONS[precision])
        assert m.sum(axis=1) == pytest.approx(_sums(psi, kb, ke, qs), rel=1e-12 if precision == "fp64" else 1e-5)
