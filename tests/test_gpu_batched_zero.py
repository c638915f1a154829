"""FP32 batches: the x = 0 transforms of all states in one launch (with states of the queue, or
from twelve larger states on) against each state's own call, whose x = 0 is a sweep of its own."""
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [[12] * 11, [12] * 12, [12, 13, 14, 15] * 3, [5, 12], [11, 16, 1, 13], [3]], ids=str)
def test_batched_equals_single_calls(ctx, hm, ns):
    psis = [rand_state(1 << n, 800 + i) for i, n in enumerate(ns)]
    vals, lost = ctx.sre_batched(psis, (2.0, 3.0), hm.HM_FP32)
    for i, p in enumerate(psis):
        v, l = ctx.sre(p, (2.0, 3.0), hm.HM_FP32)
        # the same roundings per X-string; only the FP64 sums run in another order
        assert vals[i] == pytest.approx(v, rel=1e-11, abs=1e-11)
        assert lost[i] == pytest.approx(l, abs=1e-11)


def test_ring_of_the_zero_transforms_is_what_they_need(ctx, hm, oracle):
    """The x = 0 transforms of states with a sweep of their own share a queue launch, whose ring
    holds one X-string a slot whatever the knobs say: these ask for 256 GiB, more than the GPU
    has."""
    N = hm._native
    psis = [rand_state(1 << 15, 860 + i) for i in range(12)]
    try:
        N.set_param(N.HM_PARAM_QUEUE_SLOTS, 64)
        N.set_param(N.HM_PARAM_QUEUE_SLOT_MIB, 4096)
        vals, lost = ctx.sre_batched(psis, (2.0,), hm.HM_FP32)
    finally:
        N.set_param(N.HM_PARAM_QUEUE_SLOTS, 0)
        N.set_param(N.HM_PARAM_QUEUE_SLOT_MIB, 0)
    assert vals[0][0] == pytest.approx(oracle.sre(psis[0], 2)[0], rel=1e-6)
    assert max(lost) < 1e-6
