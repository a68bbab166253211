"""Dynamic solves (FP32 matrix with FP64 vectors) of a batch in which some
instances iterate on chip and some stream, before and after autotuning, whose
FP32 and FP64 row blocks may be cut differently: every instance certifies and
the objectives agree to the tolerance (1e-6 relative, either side: 2e-6 of
1 + |objective|, and a factor 10 for the scaling of the residual to the gap)."""
import numpy as np
import pytest
from resident_worker import rows_lp

import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_dynamic_batch_with_streamed_instances_after_autotune():
    # instances 1 and 3 have rows of more than 1,024 entries, which only streaming holds
    lps = [W.random_feasible_lp(300, 751, 7, seed=1), rows_lp([1200, 4, 60, 1500] + [9] * 400, 1700, 5),
           W.random_feasible_lp(900, 2251, 7, seed=2), rows_lp([5000, 3] + [30] * 300, 6000, 6)]
    opt = gb.Options(tol=1e-6, max_iter=40_000, precision=gb.Precision.Dynamic, stall_checks=1, stall_checks_l2=200)
    with gb.BatchSolver(lps, opt) as bs:
        before = bs.solve(opt)
        bs.autotune(iters=20)
        after = bs.solve(opt)
    assert sum(r.l2_iterations for r in after) > 0
    for a, b in zip(before, after):
        assert a.status_name == b.status_name == "OPTIMAL"
        assert max(b.rel_primal, b.rel_dual, b.rel_gap) <= 1e-6 * 1.0000001
        assert abs(a.pobj - b.pobj) <= 2e-5 * (1 + abs(a.pobj))
        assert np.all(np.isfinite(b.x)) and np.all(np.isfinite(b.y))
