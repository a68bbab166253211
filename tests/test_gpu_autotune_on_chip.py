"""Autotuning an LP whose solves iterate on chip: the tuner times what a solve
runs, so it does not trade the on-chip iterations for a cut that is faster in
the streaming kernels alone.  Rows of 600 entries are STREAM rows at the default
cut of 2,048 nonzeros and LONG rows, which no cluster holds, at 512."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
CHILD = """
import sys
sys.path.insert(0, "tests")
import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W
from resident_worker import rows_lp
lps = [rows_lp([600] * 60, 3000, 1), rows_lp([600] * 30 + [5] * 200, 2000, 2), W.random_feasible_lp(300, 751, 7, seed=3)]
for lps in ([lps[0]], lps):
    for prec in ("Mixed", "Double"):
        opt = gb.Options(tol=1e-13, max_iter=512, precision=gb.Precision[prec])
        with gb.BatchSolver(lps, opt) as bs:
            a = bs.solve(opt)
            t = bs.autotune(iters=20)
            sys.stderr.write(f"case {len(lps)} {prec}\\n")
            sys.stderr.flush()
            b = bs.solve(opt)
            assert t["ms_per_iter_tuned"] <= 1.05 * t["ms_per_iter_default"] < 0.02, t
            assert t["ms_per_iter_tuned_f64"] <= 1.05 * t["ms_per_iter_default_f64"] < 0.02, t
            assert set(t["block_nnz"].tolist() + t["block_nnz_f64"].tolist()) == {2048}, t
            for x, y in zip(a, b):
                assert x.iterations == y.iterations and (x.x == y.x).all() and (x.y == y.y).all()
            sys.stderr.write("end\\n")
"""


def test_on_chip_instances_stay_on_chip():
    p = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env=dict(os.environ, GANIT_B200_TRACE="1"))
    assert p.returncode == 0, p.stderr[-2000:]
    # the solves run on plans made while tuning: none is packed again
    assert p.stderr.count("resident f32") >= 4 and p.stderr.count("resident f64") >= 4
    solves = [part.split("end\n", 1)[0] for part in p.stderr.split("case ")[1:]]
    assert len(solves) == 4 and not any("resident f" in part for part in solves)
