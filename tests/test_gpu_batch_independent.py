"""An instance that iterates on chip has the same norm, and so the same step
sizes and FP32 iterates to the bit, whatever shares its batch: next to a tiny
one it spreads over the largest cluster that its size pays for, in a crowd it
gets the fewest CTAs that hold it.  FP64 sums follow the cluster in their last
bits: 128 iterations over rows of L <= 64 entries differ by 128 (L + 6) 8 2^-53 =
8e-12 relative.  (A batch of one folds its scaling over the whole GPU, in another
order.)"""
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
tiny = W.random_feasible_lp(10, 25, 3, seed=1)
mine = [W.random_feasible_lp(m, 5 * m // 2, 7, seed=m) for m in (60, 300, 701, 1000)]
crowd = [W.random_feasible_lp(m, 2 * m, 6, seed=m) for m in range(100, 1300, 20)]
got = {}
for prec in ("Double", "Mixed"):
    opt = gb.Options(tol=1e-13, max_iter=128, precision=gb.Precision[prec])
    for name, lps, at in [(f"pair{i}", [lp, tiny], [i]) for i, lp in enumerate(mine)] + [
            ("together", mine, [0, 1, 2, 3]), ("crowd", mine + crowd, [0, 1, 2, 3])]:
        sys.stderr.write(f"case {prec} {name}\\n")
        sys.stderr.flush()
        with gb.BatchSolver(lps, opt) as bs:
            for i, r in zip(at, bs.solve(opt)):
                got[f"{prec}.{i}.{name.rstrip('0123')}"] = np.concatenate([[r.iterations, r.norm_a], r.x, r.y])
opt = gb.Options(tol=1e-13, max_iter=64)
def norms(lps):
    with gb.BatchSolver(lps, opt) as bs:
        return [r.norm_a for r in bs.solve(opt)]
got["norms.crowd"] = np.array(norms(crowd))
got["norms.pairs"] = np.array([norms([lp, tiny])[0] for lp in crowd])
np.savez(sys.argv[1], **got)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    f = str(tmp_path_factory.mktemp("ind") / "r.npz")
    p = subprocess.run([sys.executable, "-c", CHILD, f], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env=dict(os.environ, GANIT_B200_TRACE="1"))
    assert p.returncode == 0, p.stderr[-2000:]
    return dict(np.load(f)), p.stderr


def test_clusters_differ(run):
    pair, crowd = run[1].split("case Double pair3")[1], run[1].split("case Double crowd")[1]
    assert "in clusters of 16," in pair.split("case ")[0]
    assert "in clusters of 16," not in crowd.split("case ")[0]


@pytest.mark.parametrize("prec", ["Double", "Mixed"])
def test_same_in_a_pair_together_and_in_a_crowd(run, prec):
    for i in range(4):
        pair = run[0][f"{prec}.{i}.pair"]
        assert pair[0] == 128
        for other in ("together", "crowd"):
            got = run[0][f"{prec}.{i}.{other}"]
            assert got[0] == 128 and got[1] == pair[1], f"{i} {other}: norm"
            if prec == "Mixed":
                np.testing.assert_array_equal(got, pair, err_msg=f"{i} {other}")
            else:
                assert np.linalg.norm(got[2:] - pair[2:]) <= 8e-12 * np.linalg.norm(pair[2:]), f"{i} {other}"


def test_sixty_norms_in_pairs_and_in_a_crowd(run):
    np.testing.assert_array_equal(run[0]["norms.pairs"], run[0]["norms.crowd"])
