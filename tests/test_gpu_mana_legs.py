"""Mana of density matrices by passes of one to three legs (N = 1 .. 8 digits): against the
oracle, and for N = 7 and 8 through products, whose Mana is the sum of the factors'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(N, seed):
    g = np.random.default_rng(seed)
    return g.normal(size=(3 ** N, 3 ** N)) + 1j * g.normal(size=(3 ** N, 3 ** N))


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6])
def test_passes_against_oracle(ctx, oracle, N):
    m = _matrix(N, 30 + N)
    assert ctx.mana_mixed(m) == pytest.approx(oracle.mana_mixed(m), rel=1e-12)


@pytest.mark.parametrize("na,nb", [(1, 3), (2, 5), (4, 3), (3, 5)])
def test_products(ctx, na, nb):
    a, b = _matrix(na, 40 + na), _matrix(nb, 50 + nb)
    assert ctx.mana_mixed(np.kron(a, b)) == pytest.approx(ctx.mana_mixed(a) + ctx.mana_mixed(b), rel=1e-12)
