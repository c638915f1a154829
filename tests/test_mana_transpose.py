"""Mana of a density matrix does not change under transposition: A_u^T is again a phase-point
operator, so the sum of |tr(A_u rho^T)| over all u is that of |tr(A_u rho)|, for any
matrix.  The Python layer passes a row-major matrix as it is on that ground."""
import numpy as np
import pytest


def _matrix(N, seed):
    g = np.random.default_rng(seed)
    return g.normal(size=(3 ** N, 3 ** N)) + 1j * g.normal(size=(3 ** N, 3 ** N))  # not Hermitian


@pytest.mark.parametrize("N", [1, 2, 3])
def test_oracle_value_is_that_of_the_transpose(oracle, N):
    m = _matrix(N, N)
    assert oracle.mana_mixed(np.ascontiguousarray(m.T)) == pytest.approx(oracle.mana_mixed(m), rel=1e-14)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [1, 2, 4])
def test_every_memory_order(ctx, hm, oracle, N):
    m = _matrix(N, 10 + N)
    big = np.zeros((2 * 3 ** N, 2 * 3 ** N), dtype=complex)
    big[::2, ::2] = m
    ref = oracle.mana_mixed(m)
    for r in (np.ascontiguousarray(m), np.asfortranarray(m), big[::2, ::2], m.T.copy().T):
        assert ctx.mana_mixed(r) == pytest.approx(ref, rel=1e-10)
        assert hm.Mana(hm.DensityMatrix(r, q=3)) == pytest.approx(ref, rel=1e-10)


@pytest.mark.gpu
def test_brick_wall_in_place_forms(hm):
    gates = [hm.haar_random_unitary(2, 2, np.random.default_rng(i)) for i in range(len(hm.brick_wall_pairs(6, 3)))]
    v = np.zeros(64, dtype=complex)
    v[0] = 1.0
    sv = hm.StateVec(v)
    held = sv.data
    hm.apply_brick_wall(sv, 3, gates)
    assert sv.data is held
    strided = hm.StateVec(v)
    strided.data = np.zeros(128, dtype=complex)[::2]
    strided.data[:] = v
    hm.apply_brick_wall(strided, 3, gates)
    assert np.array_equal(strided.data, held)
    before = held.copy()
    with pytest.raises(hm.ArgumentError):
        hm.apply_brick_wall(sv, 3, gates[:-1])
    assert np.array_equal(held, before)
