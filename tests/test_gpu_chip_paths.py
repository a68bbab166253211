"""That the cases of the on-chip tests run where those tests say: the QPs of
qp_chip_worker.py in k_qp_chip (a rank too large for its FP64 form streams), the
systems of test_gpu_minres_chip.py in k_mr_solve_chip with one or two rows a
thread or in k_mr_solve, and the batches of test_gpu_resident_waves.py, in FP64,
in clusters of the size that their line gives or streaming.  The paths are read
from the trace, which is on per process: hence the children."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HEAD = """
import sys
sys.path.insert(0, "tests")
import numpy as np
import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W
def case(name):
    sys.stderr.write(f"case {name}\\n")
    sys.stderr.flush()
"""
QP = HEAD + """
from qp_chip_worker import cases
for name, lp in [*cases(), ("rank_100", W.portfolio_qp(60_000, 100, seed=1))]:
    for prec in ("Mixed", "Double"):
        case(f"{name}.{prec}")
        gb.solve_pdhg_gpu(lp, gb.Options(tol=1e-13, max_iter=5, check_every=5, precision=gb.Precision[prec]))
"""
MINRES = HEAD + """
opt = gb.Options(tol=1e-6, precision=gb.Precision.Mixed)
for shapes in ([(3, 7, 2)], [(40, 90, 5), (60, 130, 6)], [(520, 1100, 10), (30, 61, 4)], [(600, 1300, 8), (200, 420, 10)],
               [(1250, 2600, 14)]):
    lps = [W.nondegenerate_lp(m, n, k, seed=9000 + i, max_cond=5e4) for i, (m, n, k) in enumerate(shapes)]
    rows = max(max(int(np.sum(lp.meta["interior"])), int(np.sum(lp.meta["tight"]))) for lp in lps)
    case(rows)
    ds = gb.DiffSolver(lps, opt, tail_iters=40, ckpt_every=10)
    ds.forward(opt)
    ds.backward(np.ones(int(ds.n_off[-1])), np.ones(int(ds.m_off[-1])))
    ds.close()
"""
WAVES = HEAD + """
from test_gpu_resident_waves import SHAPES
opt = gb.Options(tol=1e-13, max_iter=64)
for n, m, density, count in SHAPES:
    lp = W.milp_node(n=n, knapsacks=m, density=density, up_blocked=0, down_blocked=0, seed=3)
    case(f"{n} {count}")
    gb.BatchSolver([lp] * count, opt).close()
"""


def parts(code):
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env=dict(os.environ, GANIT_B200_TRACE="1"))
    assert p.returncode == 0, p.stderr[-2000:]
    return dict(part.split("\n", 1) for part in p.stderr.split("case ")[1:])


def test_qps_run_on_chip():
    got = parts(QP)
    assert len(got) == 24
    for name, trace in got.items():
        levels = set(re.findall(r"qp on chip (f\d\d/f\d\d)", trace))
        if name.startswith("rank_100"):
            assert "f64/f64" not in levels, name
        else:
            assert levels >= {"f64/f64" if name.endswith("Double") else "f32/f32"}, name
    kept = re.search(r"f64/f64: (\d+) of 169 columns", got["budget_100000_50.Double"])
    assert 0 < int(kept.group(1)) < 169  # the rest from L2


def test_minres_runs_in_the_form_of_its_size():
    got = parts(MINRES)
    forms = [set(re.findall(r"minres on chip: \d+ rows, (\d) a thread", t)) for t in got.values()]
    for rows, form in zip(map(int, got), forms):
        assert form == ({"1"} if rows <= 512 else {"2"} if rows <= 1024 else set()), (rows, form)
    assert {frozenset(f) for f in forms} == {frozenset("1"), frozenset("2"), frozenset()}


def test_batches_take_the_clusters_of_their_line():
    got = {k: set(re.findall(r"resident f64: \d+ CTAs in clusters of (\d+)", t)) for k, t in parts(WAVES).items()}
    assert got == {"10000 7": {"16"}, "10000 8": set(), "7500 30": {"8"}, "7500 31": set(), "5000 15": {"8"},
                   "5000 16": {"4"}}
