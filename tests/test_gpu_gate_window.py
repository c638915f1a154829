"""Brick walls in windows of sites (csrc/stateprep.cu): sizes around the tile of one CTA (9 to
12 qubits, 6 or 7 qutrits), windows at both ends, more gates than a pass holds, random (not
unitary) gates.  Every gate's arithmetic is that of the one-gate kernel; while the whole
state is one tile the gates also keep their order, so the result equals hm_apply_2gate
gate by gate to the bit.  Above that, gates on disjoint sites change places (they commute
in exact arithmetic only) and the oracle's bound alone holds."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,depth", [(2, 2, 3), (2, 3, 4), (2, 9, 70), (2, 10, 5), (2, 11, 9), (2, 12, 60), (2, 13, 9), (2, 14, 1),
                                       (2, 15, 41), (2, 18, 6), (2, 19, 3), (2, 20, 2),
                                       (3, 2, 3), (3, 6, 5), (3, 7, 9), (3, 8, 7),
                                       (3, 9, 12), (3, 10, 3)])
def test_windows_equal_single_gates(hm, ctx, oracle, q, n, depth):
    rng = np.random.default_rng(100 * n + depth)
    pairs = hm.brick_wall_pairs(n, depth)
    gates = [(rng.normal(size=(q * q, q * q)) + 1j * rng.normal(size=(q * q, q * q))) / (1.4 * q) for _ in pairs]
    psi = rand_state(q ** n, 30 + n)
    out = ctx.brick_wall(psi, q, depth, gates)
    if n <= (9 if q == 2 else 7):
        ref = psi
        for g, (s1, s2) in zip(gates, pairs):
            ref = ctx.apply_2gate(ref, q, g, s1, s2)
        assert np.array_equal(out, ref)
    o = oracle.brick_wall(psi, q, depth, gates)
    assert np.abs(out - o).max() <= 1e-11 * np.abs(o).max()
