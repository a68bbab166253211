"""Child process of tests/test_gpu_grid.py: a fixed number of iterations of LPs
too large for one cluster, points written to the given npz file.
GANIT_B200_RESIDENT is read once per process, hence the child."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import ganit_v2_b200 as gb  # noqa: E402
from ganit_v2_b200 import workloads as W  # noqa: E402
from tests.resident_worker import rows_lp  # noqa: E402


def cases():
    yield "blend_all_on_chip", W.blending_lp(20, 8, 4, 100, seed=3)
    yield "blend_part_in_l2", W.blending_lp(60, 16, 5, 365, seed=1)  # FP32: 60 % on chip; FP64 streams
    yield "random_scattered", W.random_feasible_lp(6000, 15_001, 12, seed=2)
    yield "few_long_rows", rows_lp([1024] * 140 + [0, 3], 20_011, 4)  # shares of one row, and an empty one
    yield "many_short_rows", rows_lp([2] * 70_000 + [0] * 5 + [31], 900, 5)  # positions beyond 16 bits
    yield "long_row_streams", rows_lp([1100] + [20] * 9000, 5000, 6)


def main(out):
    got = {}
    for name, lp in cases():
        for prec in ("Mixed", "Dynamic", "Double", "MixedBf16"):
            for ce, it in ((32, 64), (3, 3)):
                opt = gb.Options(tol=1e-13, max_iter=it, check_every=ce, precision=gb.Precision[prec])
                r = gb.solve_pdhg_gpu(lp, opt)
                got[f"{name}.{prec}.{ce}"] = np.concatenate([[r.iterations], r.x, r.y])
    np.savez(out, **got)


if __name__ == "__main__":
    main(sys.argv[1])
