"""Gradients of the sizes whose X-strings one warp holds (n <= 11): every register split, the
run-time power, the gather with fewer entries than a block and with one or several splits."""
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [1, 2, 3, 8])
@pytest.mark.parametrize("n", range(1, 12))
def test_grad_one_warp_sizes(ctx, oracle, n, q):
    psi = rand_state(1 << n, 700 + n)
    v, g = ctx.sre_grad(psi, q)
    ov, og = oracle.sre_grad(psi, q)
    assert abs(v - ov) <= 1e-10 * max(1.0, abs(ov))  # q = 1: the value is 0 up to rounding
    assert abs(g - og).max() <= 1e-10 * abs(og).max()
