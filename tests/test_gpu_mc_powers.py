"""MC_SRE with Renyi indices whose powers come from pow(), for which the evaluating warps stage
their values in shared memory, and with half-integers from registers.  Same
bounds as test_gpu_mc_mana_grad.py: accepted masks bit-exact, estimates within 1e-10 relative."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


def check(ctx, hm, oracle, n, nb, ns, q):
    psi = rand_state(1 << n, 640 + n)
    pd, rs = hm.proposal_stream(n, nb, ns, seed=19)
    pd[0, 0] = 0  # a zero proposal is never accepted
    m2, M2, M2ADD, P2, masks = ctx.mc_sre(psi, q, nb, ns, pd, rs)
    om2, oM2, oM2ADD, oP2 = oracle.mc_sre(psi, q, nb, ns, pd, rs)
    assert m2 == pytest.approx(om2, rel=1e-10)
    assert np.allclose(M2, oM2, rtol=1e-10) and np.allclose(M2ADD, oM2ADD, rtol=1e-10)
    assert np.allclose(P2, oP2, rtol=1e-10)
    for i in range(0, nb, max(1, nb // 5)):
        _, om = oracle.mc_sre_beta(psi, q, i / (nb - 1), pd[i], rs[i])
        assert int(masks[i]) == int(om[-1])


@pytest.mark.parametrize("n,nb,ns,q", [(16, 65, 3, 2.7), (17, 17, 3, 2.7), (17, 17, 3, 3.5), (18, 5, 4, 2.7),
                                       (19, 3, 3, 2.7), (20, 3, 2, 2.7), (21, 3, 2, 2.7), (21, 3, 2, 15.5)])
def test_step_kernels(ctx, hm, oracle, n, nb, ns, q):
    check(ctx, hm, oracle, n, nb, ns, q)


@pytest.mark.parametrize("n,nb,ns,q", [(3, 3, 12, 2.7), (8, 5, 20, 2.7), (11, 3, 12, 2.7), (12, 3, 8, 2.7),
                                       (13, 3, 8, 2.7), (14, 5, 6, 2.7), (14, 75, 2, 2.7), (15, 3, 6, 2.7),
                                       (15, 19, 3, 2.7), (16, 3, 5, 2.7), (17, 3, 4, 2.7)])
def test_chains_of_one_launch(ctx, hm, oracle, n, nb, ns, q):
    """One warp, one CTA, and clusters of two, four and eight CTAs to a chain: the staged values
    share their memory with the exchange of the chain's other warps."""
    check(ctx, hm, oracle, n, nb, ns, q)
