"""Pass 2 of the two-pass sweeps drops the L2 lines that it has read, and pass 1 of the stage
after next rewrites them.  Tiny batches make the stages short, so that a late drop would meet
the new rows: every repetition has to give the same bits, and the sums those of the queue
sweep, which drops nothing.  Every kernel and layout that drops lines: k_sre_wide_stage with all
rows of a column in registers (n <= 17), with rows on lane bits (n >= 18), with units
paired to whole lines (FP64 n = 21, FP32 n = 20, 21), and k_sre_stage (FP64 n = 19 with q = 2 and
3, n = 20)."""
import numpy as np
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu

Q2, Q23 = (2.0,), (2.0, 3.0)


@pytest.mark.parametrize("graph", [0, 8], ids=["direct", "replayed"])
@pytest.mark.parametrize("n,precision,qs,X", [
    (15, "fp64", Q2, 1), (16, "fp64", Q2, 3), (17, "fp64", Q2, 1), (18, "fp64", Q2, 1), (18, "fp64", Q23, 2),
    (19, "fp64", Q2, 1), (19, "fp64", Q23, 1), (20, "fp64", Q2, 1), (20, "fp64", Q23, 2), (20, "fp64", (4.0,), 1),
    (21, "fp64", Q2, 1), (21, "fp64", Q23, 2),
    (16, "fp32", Q2, 1), (18, "fp32", Q2, 1), (19, "fp32", Q2, 2), (20, "fp32", Q2, 1), (21, "fp32", Q2, 1),
    (21, "fp32", (2.7,), 1)])
def test_repetitions_are_bit_identical(ctx, hm, n, precision, qs, X, graph):
    N, p = hm._native, hm.PRECISIONS[precision]
    psi = rand_state(1 << n, 1900 + n)
    kb, ke = (1 << (n - 1)) - 11, (1 << (n - 1)) + 40 * X + 1
    try:
        N.set_param(N.HM_PARAM_ENGINE, 1)
        N.set_param(N.HM_PARAM_BATCH, X)
        N.set_param(N.HM_PARAM_GRAPH, graph)
        first = ctx.sre_range(psi, kb, ke, qs, p)
        for _ in range(12):
            again = ctx.sre_range(psi, kb, ke, qs, p)
            assert np.array_equal(again[0], first[0]) and np.array_equal(again[1], first[1])
        N.set_param(N.HM_PARAM_ENGINE, 2)
        p2, m = ctx.sre_range(psi, kb, ke, qs, p)
    finally:
        N.set_param(N.HM_PARAM_BATCH, 0)
        N.set_param(N.HM_PARAM_GRAPH, 0)
        N.set_param(N.HM_PARAM_ENGINE, 0)
    # the bounds used between the engines in test_gpu_wide.py
    tol = 1e-13 if precision == "fp64" else 1e-6
    assert first[0].sum() == pytest.approx(p2.sum(), rel=tol)
    assert first[1].sum(axis=1) == pytest.approx(m.sum(axis=1), rel=tol)
