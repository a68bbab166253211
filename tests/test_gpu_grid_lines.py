"""Single LPs on both sides of the lines where one LP is kept by the whole GPU
or streams: FP32 with under four rows per CTA (592), and FP64 matrices that fit
only in part and gather more entries than they hold.  GANIT_B200_RESIDENT is
read once per process, hence the children.  FP32 iterates keep their bits; 32
FP64 iterations over rows of L <= 1024 entries differ by 32 (L + 6) 8 2^-53 =
2.9e-11 relative between two orders of summation."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHILD = """
import sys
import numpy as np
import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W
kind, rows, prec, out = sys.argv[1], int(sys.argv[2]), sys.argv[3], sys.argv[4]
if kind == "node":
    lp = W.milp_node(n=30000, knapsacks=rows, density=0.01, up_blocked=0, down_blocked=0, seed=1)
else:
    lp = W.random_feasible_lp(rows, 30000, 30, seed=7)
r = gb.solve_pdhg_gpu(lp, gb.Options(tol=1e-13, max_iter=32, check_every=32, precision=gb.Precision[prec]))
np.save(out, np.concatenate([[r.iterations], r.x, r.y]))
"""


@pytest.mark.parametrize("kind, rows, prec, on_chip", [
    ("node", 591, "Mixed", False), ("node", 592, "Mixed", True), ("node", 591, "Double", True),
    ("random", 20000, "Double", False), ("random", 20000, "Mixed", True)])
def test_either_side_of_a_line_ends_in_the_same_point(tmp_path, kind, rows, prec, on_chip):
    got = []
    for on in ("1", "0"):
        f = str(tmp_path / f"r{on}.npy")
        p = subprocess.run([sys.executable, "-c", CHILD, kind, str(rows), prec, f], capture_output=True, text=True,
                           timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                           env=dict(os.environ, GANIT_B200_RESIDENT=on, GANIT_B200_TRACE="1"))
        assert p.returncode == 0, p.stderr[-2000:]
        assert (f"grid f{32 if prec == 'Mixed' else 64}" in p.stderr) == (on_chip and on == "1")
        got.append(np.load(f))
    if prec == "Mixed":
        np.testing.assert_array_equal(got[0], got[1])
    else:
        assert np.linalg.norm(got[0] - got[1]) <= 2.9e-11 * np.linalg.norm(got[1])
