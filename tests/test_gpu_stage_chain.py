"""The chained stages of a sweep: direct launches up to one graph's worth of stages, replays of a
captured graph above that, which end with stages that have no batch."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,qs", [(15, (2.0,)), (18, (2.0, 3.0)), (20, (2.0,)), (22, (2.0,))])
def test_direct_launches_and_replays_agree(ctx, hm, n, qs):
    N = hm._native
    psi, kb, ke = rand_state(1 << n, 150 + n), 2000, 2040
    extra = 2 if n == 22 else 1  # stages after the last batch's first pass
    try:
        N.set_param(N.HM_PARAM_BATCH, 1)
        direct = ctx.sre_range(psi, kb, ke, qs, hm.HM_FP64)
        assert ctx.last_launch_count() == 40 + extra + 1  # the stages and the fold
        N.set_param(N.HM_PARAM_GRAPH, 16)
        replay = ctx.sre_range(psi, kb, ke, qs, hm.HM_FP64)
        assert ctx.last_launch_count() == 3 * 17 + 1
    finally:
        N.set_param(N.HM_PARAM_BATCH, 0)
        N.set_param(N.HM_PARAM_GRAPH, 0)
    assert np.array_equal(direct[0], replay[0]) and np.array_equal(direct[1], replay[1])
