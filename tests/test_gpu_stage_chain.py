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


def test_default_batch_belongs_to_the_kernel(ctx, hm):
    """At n = 20 in FP64 q = 2 and other q run different kernels, whose default batches are 10 and
    9: 90 X-strings take 9 and 10 batches, one stage more, and the fold."""
    psi = rand_state(1 << 20, 170)
    counts = []
    for qs in ((2.0,), (4.0,)):
        ctx.sre_range(psi, 2000, 2090, qs, hm.HM_FP64)
        counts.append(ctx.last_launch_count())
    assert counts == [11, 12]
