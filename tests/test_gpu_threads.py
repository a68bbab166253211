"""Problems solved from several threads at once, each in its own stream: the
cooperative kernels that wait for words of their own other CTAs (k_grid,
k_qp_chip) and the clusters (k_resident) share the GPU with one another, and
every solve gives the bits that it gives alone."""
import threading

import numpy as np
import pytest

import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_solves_in_threads_give_the_bits_they_give_alone():
    lps = [W.blending_lp(60, 16, 5, 26, seed=1), W.blending_lp(60, 16, 5, 30, seed=2), W.portfolio_qp(8009, 33, seed=3),
           W.random_feasible_lp(2000, 5000, 8, seed=4)]
    opts = [gb.Options(tol=1e-13, max_iter=512, precision=p)
            for p in (gb.Precision.Double, gb.Precision.Mixed, gb.Precision.Mixed, gb.Precision.Double)]
    problems = [gb.Problem(lp, o) for lp, o in zip(lps, opts)]
    alone = [p.solve(o) for p, o in zip(problems, opts)]
    got, errors = [[] for _ in lps], []

    def run(k):
        try:
            for _ in range(6):
                got[k].append(problems[k].solve(opts[k]))
        except Exception as e:
            errors.append(f"{k}: {e}")

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(lps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and not any(t.is_alive() for t in threads)
    for a, rs in zip(alone, got):
        assert len(rs) == 6
        for r in rs:
            assert r.iterations == a.iterations
            np.testing.assert_array_equal(r.x, a.x)
            np.testing.assert_array_equal(r.y, a.y)
    for p in problems:
        p.close()
