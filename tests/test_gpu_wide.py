"""The sweep kernels of csrc/sre_wide.cuh against the queue sweep, which transforms the same
X-strings by the two-pass route: sub-ranges of the Gray codes that are ragged, start past 0
or hold a single X-string, every moment set, both precisions.

FP64 sums are added from different operation orders of ~20 roundings per value; the
averaging over 2^n values keeps the difference near 1e-16, 1e-13 is the bound used between
the engines elsewhere.  FP32 is held to the precision's stated 1e-6."""
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu

QS = {"q2": (2.0,), "q23": (2.0, 3.0), "gen": (4.0, 2.5, 1.0)}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("qs", sorted(QS))
@pytest.mark.parametrize("n", [12, 13, 14])
def test_single_cta_ranges(ctx, hm, n, qs, precision):
    N = hm._native
    psi = rand_state(1 << n, 900 + n)
    full = 1 << n
    tol = 1e-13 if precision == "fp64" else 1e-6
    for kb, ke in [(0, 1), (0, 150), (1, 2), (700, 1333), (full - 37, full)]:
        p2, m = ctx.sre_range(psi, kb, ke, QS[qs], hm.PRECISIONS[precision])
        try:
            N.set_param(N.HM_PARAM_ENGINE, 2)
            p2r, mr = ctx.sre_range(psi, kb, ke, QS[qs], hm.PRECISIONS[precision])
        finally:
            N.set_param(N.HM_PARAM_ENGINE, 0)
        assert p2.sum() == pytest.approx(p2r.sum(), rel=tol)
        assert m.sum(axis=1) == pytest.approx(mr.sum(axis=1), rel=tol)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("qs", sorted(QS))
@pytest.mark.parametrize("n", [15, 16, 17, 18, 19, 20, 21])
def test_two_pass_ranges(ctx, hm, n, qs, precision):
    N = hm._native
    psi = rand_state(1 << n, 900 + n)
    full = 1 << n
    tol = 1e-13 if precision == "fp64" else 1e-6
    ranges = [(0, 1), (0, 5), (1021, 1034)] if n >= 19 else [(0, 1), (0, 150), (1, 2), (3000, 3333), (full - 37, full)]
    for kb, ke in ranges:
        p2, m = ctx.sre_range(psi, kb, ke, QS[qs], hm.PRECISIONS[precision])
        try:
            N.set_param(N.HM_PARAM_BATCH, 3)  # several stages, the last one not full
            p2s, ms = ctx.sre_range(psi, kb, ke, QS[qs], hm.PRECISIONS[precision])
            N.set_param(N.HM_PARAM_BATCH, 0)
            N.set_param(N.HM_PARAM_ENGINE, 2)
            p2r, mr = ctx.sre_range(psi, kb, ke, QS[qs], hm.PRECISIONS[precision])
        finally:
            N.set_param(N.HM_PARAM_BATCH, 0)
            N.set_param(N.HM_PARAM_ENGINE, 0)
        for p, v in ((p2, m), (p2s, ms)):
            assert p.sum() == pytest.approx(p2r.sum(), rel=tol)
            assert v.sum(axis=1) == pytest.approx(mr.sum(axis=1), rel=tol)


@pytest.mark.parametrize("n,q", [(12, 4), (13, 1), (13, 3), (14, 8)])
def test_grad_single_cta(ctx, oracle, n, q):
    psi = rand_state(1 << n, 950 + n)
    v, g = ctx.sre_grad(psi, q)
    ov, og = oracle.sre_grad(psi, q)
    assert abs(v - ov) <= 1e-10 * max(1.0, abs(ov))  # q = 1: the value is 0 up to rounding
    assert abs(g - og).max() <= 1e-10 * abs(og).max()


@pytest.mark.parametrize("L", [1, 2, 3, 5, 7, 8])
def test_mana_pairs_equal_single_x_strings(ctx, L):
    # X-strings of a range share transforms in pairs; a range of one has no partner
    psi, D = rand_state(3 ** L, 970 + L), 3 ** L
    for a, b in {(0, D), (D // 3, D), (max(0, D - 41), D)}:
        if b - a <= 300:
            singles = sum(ctx.mana_pure_range(psi, x, x + 1).sum() for x in range(a, b))
            assert ctx.mana_pure_range(psi, a, b).sum() == pytest.approx(singles, rel=1e-13)
