"""A batch whose later state cannot be launched: the call reports the error with nothing of the
earlier states' sweeps still in flight, and the context stays usable."""
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu

CUDA_STREAM_LEGACY = 1  # cudaStreamLegacy: runs kernels, refuses graph capture


def test_failed_batch_leaves_nothing_in_flight(hm, oracle):
    import torch
    ctx = hm._native.Context(0)
    legacy = torch.cuda.default_stream()
    assert legacy.query()  # torch is set up here, not while the sweeps run
    large = rand_state(1 << 16, 60)
    # the large sweep replays a captured graph; its buffers are there before the failing call
    ref, _ = ctx.sre(large, (2.0,), hm.HM_FP64)
    small = [rand_state(1 << 14, 61 + i) for i in range(3)]
    try:
        ctx.set_stream(CUDA_STREAM_LEGACY)
        with pytest.raises(hm.HadaMAGError):
            ctx.sre_batched(small * 13 + [large], (2.0,), hm.HM_FP64)  # 39 sweeps of 0.5 ms before it
        assert legacy.query()
    finally:
        ctx.set_stream(0)
    for precision, tol in ((hm.HM_FP32, 1e-6), (hm.HM_FP64, 1e-10)):
        vals, lost = ctx.sre_batched(small + [large], (2.0,), precision)
        for p, v in zip(small + [large], vals):
            assert v[0] == pytest.approx(ref[0] if p is large else oracle.sre(p, 2)[0], rel=tol)
        assert max(lost) < 1e-6
