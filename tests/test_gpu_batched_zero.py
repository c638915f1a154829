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
