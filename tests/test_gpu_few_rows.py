"""LPs of few rows and many columns, or the reverse, on chip in clusters with
more CTAs than the smaller side has slices, against the streaming kernels
(GANIT_B200_RESIDENT=0, read once per process, hence the children): Mixed
iterates keep their bits; 128 FP64 iterations over rows of L <= 1024 entries
differ by 128 (L + 6) 8 2^-53 = 1.2e-10 relative between two orders of
summation; the norm (50 steps, each a sum over a row and one over at most 6,000
columns) by 50 * 7,030 * 1.1e-16 = 3.9e-11."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
CHILD = """
import sys
import numpy as np
sys.path.insert(0, "tests")
import ganit_v2_b200 as gb
from resident_worker import rows_lp
got = {}
rng = np.random.default_rng(0)
for name, lens, n in (("ten_rows", [900] * 10, 5000), ("two_rows", [1000, 31], 2000), ("seven_rows", [1024, 5, 1, 33, 32, 31, 65], 1500),
                      ("few_columns", rng.integers(1, 3, size=6000).tolist(), 11)):
    for prec in ("Mixed", "Double"):
        opt = gb.Options(tol=1e-13, max_iter=128, precision=gb.Precision[prec])
        r = gb.solve_pdhg_gpu(rows_lp(lens, n, 7), opt)
        got[f"{name}.{prec}"] = np.concatenate([[r.iterations, r.norm_a], r.x, r.y])
np.savez(sys.argv[1], **got)
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for on in ("1", "0"):
        f = str(tmp_path_factory.mktemp("few") / f"r{on}.npz")
        p = subprocess.run([sys.executable, "-c", CHILD, f], capture_output=True, text=True, timeout=300,
                           cwd=os.path.dirname(HERE), env=dict(os.environ, GANIT_B200_RESIDENT=on, GANIT_B200_TRACE="1"))
        assert p.returncode == 0, p.stderr[-2000:]
        out.append((dict(np.load(f)), p.stderr))
    return out


def test_every_case_ran_in_a_cluster(both):
    # every problem makes an FP64 plan, the Mixed ones an FP32 plan too
    assert both[0][1].count("resident f64") == 8 and both[0][1].count("resident f32") == 4
    assert "in clusters of 16," in both[0][1] and "in clusters of 8," in both[0][1]
    assert "resident f" not in both[1][1]


@pytest.mark.parametrize("name", ["ten_rows", "two_rows", "seven_rows", "few_columns"])
def test_iterates_match_streamed_ones(both, name):
    for prec in ("Mixed", "Double"):
        on, off = both[0][0][f"{name}.{prec}"], both[1][0][f"{name}.{prec}"]
        assert on[0] == off[0] == 128
        assert abs(on[1] - off[1]) <= 3.9e-11 * off[1]
        if prec == "Mixed":
            np.testing.assert_array_equal(on[2:], off[2:])
        else:
            assert np.linalg.norm(on[2:] - off[2:]) <= 1.2e-10 * np.linalg.norm(off[2:])
