"""Child process of tests/test_gpu_resident.py: a fixed number of iterations of
LPs that the on-chip kernel takes at every cluster size (and of batches where
one instance streams), points written to the given npz file.
GANIT_B200_RESIDENT is read once per process, hence the child."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import ganit_v2_b200 as gb  # noqa: E402
from ganit_v2_b200 import workloads as W  # noqa: E402
from ganit_v2_b200.lp import LP, Csr  # noqa: E402


def rows_lp(lens, n, seed):
    """LP with rows of the given lengths (some may be empty) over n boxed columns."""
    rng = np.random.default_rng(seed)
    idx = np.concatenate([rng.choice(n, size=k, replace=False) for k in lens] + [np.zeros(0, dtype=int)])
    ptr = np.concatenate([[0], np.cumsum(lens)])
    A = Csr(len(lens), n, ptr, idx, rng.standard_normal(len(idx)))
    b = rng.uniform(1.0, 2.0, size=len(lens))
    return LP(A, rng.standard_normal(n), -np.ones(n), np.ones(n), -b, b)


def cases():
    yield "one_by_one", [rows_lp([1], 1, 0)]
    yield "empty_rows", [rows_lp([0, 3, 0, 7, 1, 0], 9, 1)]
    yield "longest_row", [rows_lp([1024, 5, 1, 33, 32, 31, 65], 1500, 2)]
    yield "long_row_streams", [rows_lp([1025, 5, 9], 1500, 3)]
    for m in (50, 130, 300, 701, 1500, 3000):  # clusters of 1 to 16
        yield f"random_{m}", [W.random_feasible_lp(m, 5 * m // 2 + 1, 7, seed=m)]
    yield "wide", [rows_lp([900] * 40, 9001, 4)]
    yield "batch", [W.random_feasible_lp(m, 2 * m + 3, 6, seed=m) for m in (20, 45, 333, 900, 2500)] + [
        rows_lp([1200, 4, 60], 1400, 5), rows_lp([2] * 700, 40, 6)]


def main(out):
    got = {}
    for name, lps in cases():
        for prec in ("Mixed", "Dynamic", "Double", "MixedBf16"):
            for ce, it in ((64, 128), (5, 15), (1, 1)):
                opt = gb.Options(tol=1e-13, max_iter=it, check_every=ce, precision=gb.Precision[prec])
                with gb.BatchSolver(lps, opt) as bs:
                    for k, r in enumerate(bs.solve(opt)):
                        got[f"{name}.{prec}.{ce}.{k}"] = np.concatenate([[r.iterations], r.x, r.y])
                        got[f"norm.{name}.{k}"] = np.array([r.norm_a])
    np.savez(out, **got)


if __name__ == "__main__":
    main(sys.argv[1])
