"""Batches of instances that fill whole clusters, on both sides of the line
where a batch takes smaller clusters or streams: every instance ends where it
does alone.  128 FP64 iterations over rows of L <= 1024 entries differ by
128 (L + 6) 8 2^-53 = 1.2e-10 relative between two orders of summation; an
FP32 step size may round the other way when the norm's last bits differ:
128 * 8 * 2^-24 = 6.1e-5."""
import numpy as np
import pytest

import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu
SHAPES = [(10000, 500, 0.01, 7), (10000, 500, 0.01, 8),  # clusters of 16: one wave, more
          (7500, 200, 0.01, 30), (7500, 200, 0.01, 31),  # clusters of 8: two waves, more
          (5000, 200, 0.02, 15), (5000, 200, 0.02, 16)]  # clusters of 8 or 4


@pytest.mark.parametrize("n, m, density, count", SHAPES)
@pytest.mark.parametrize("prec, bound", [("Double", 1.2e-10), ("Mixed", 6.1e-5)])
def test_instances_of_a_batch_end_where_they_do_alone(n, m, density, count, prec, bound):
    lp = W.milp_node(n=n, knapsacks=m, density=density, up_blocked=0, down_blocked=0, seed=3)
    opt = gb.Options(tol=1e-13, max_iter=128, precision=gb.Precision[prec])
    with gb.BatchSolver([lp], opt) as bs:
        one = bs.solve(opt)[0]
    with gb.BatchSolver([lp] * count, opt) as bs:
        got = bs.solve(opt)
    assert len(got) == count
    for r in got:
        assert r.iterations == one.iterations == 128
        for a, b in ((r.x, one.x), (r.y, one.y)):
            assert np.linalg.norm(a - b) <= bound * np.linalg.norm(b)
            np.testing.assert_array_equal(a, got[0].x if a is r.x else got[0].y)
