"""What an on-chip plan needs only while it is packed is given back as soon as
the packing is done: the pinned sources of its copies and, for an LP kept by the
whole GPU, a bitmap and running counts of the gathered vectors per CTA (8 bytes
x 148 CTAs x a word per 32 rows and columns) -- at set-up, and again when the
autotuner's last plan is packed by the next solve.  The trace is read once per
process, hence the child."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
CHILD = """
import sys
import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W
opt = gb.Options(tol=1e-13, max_iter=64, precision=gb.Precision.Mixed)
for lp in (W.blending_lp(60, 16, 5, 52, seed=1), W.random_feasible_lp(300, 751, 7, seed=1)):
    sys.stderr.write(f"create {lp.m} {lp.n}\\n")
    sys.stderr.flush()
    with gb.Problem(lp, opt) as p:
        p.solve(opt)
        p.autotune(5)
        sys.stderr.write("tuned\\n")
        sys.stderr.flush()
        p.solve(opt)
"""


def test_packing_scratch_does_not_outlive_the_packing():
    p = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env=dict(os.environ, GANIT_B200_TRACE="1"))
    assert p.returncode == 0, p.stderr[-2000:]
    for part in p.stderr.split("create ")[1:]:
        m, n = (int(v) for v in part.split("\n", 1)[0].split())
        setup, later = part.split("phases", 1)[0], part.split("tuned\n", 1)[1]
        grids = setup.count("grid f")
        words = -(-m // 32) + -(-n // 32)
        back = re.findall(r"plan scratch given back: (\d+) pinned blocks, (\d+) B", setup)
        assert len(back) == 1 and int(back[0][0]) >= 1
        assert int(back[0][1]) >= grids * 8 * 148 * words
        assert "resident f" in setup if m == 300 else grids == 2
        assert "plan scratch given back" in later
