"""MC_SRE where one launch runs whole chains (csrc/mc.cu): one warp, one CTA and one cluster
per chain, more chains than fit the GPU at once, and both sides of the rule that hands
many chains to the step kernels.  Same bounds as test_gpu_mc_mana_grad.py: accepted masks
bit-exact, estimates within 1e-10 relative."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb,ns,q", [(1, 3, 20, 2), (2, 3, 40, 2), (8, 5, 60, 2), (12, 601, 2, 2), (13, 3, 40, 2),
                                       (13, 3, 10, 2.5), (14, 5, 30, 2), (14, 75, 4, 2), (15, 19, 12, 2),
                                       (15, 3, 10, 3), (16, 21, 10, 2), (16, 65, 3, 2), (17, 5, 10, 2),
                                       (17, 5, 4, 2.5), (17, 25, 3, 2)])
def test_chains_match_oracle(ctx, hm, oracle, n, nb, ns, q):
    psi = rand_state(1 << n, 600 + n)
    pd, rs = hm.proposal_stream(n, nb, ns, seed=9)
    pd[0, 0] = 0  # a zero proposal is never accepted
    m2, M2, M2ADD, P2, masks = ctx.mc_sre(psi, q, nb, ns, pd, rs)
    om2, oM2, oM2ADD, oP2 = oracle.mc_sre(psi, q, nb, ns, pd, rs)
    assert m2 == pytest.approx(om2, rel=1e-10)
    assert np.allclose(M2, oM2, rtol=1e-10) and np.allclose(M2ADD, oM2ADD, rtol=1e-10)
    assert np.allclose(P2, oP2, rtol=1e-10)
    for i in range(0, nb, max(1, nb // 5)):
        _, om = oracle.mc_sre_beta(psi, q, i / (nb - 1), pd[i], rs[i])
        assert int(masks[i]) == int(om[-1])
    lo, hi = nb // 3, nb // 3 + 2
    part = ctx.mc_sre_chains(psi, q, nb, lo, hi, ns, pd[lo:hi], rs[lo:hi])
    assert np.array_equal(part[0], M2[lo:hi]) and np.array_equal(part[3], masks[lo:hi])
