"""Child process of tests/test_gpu_qp_chip.py: a fixed number of iterations of
diagonal-plus-low-rank QPs, points written to the given npz file.
GANIT_B200_RESIDENT is read once per process, hence the child."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import ganit_v2_b200 as gb  # noqa: E402
from ganit_v2_b200 import workloads as W  # noqa: E402
from ganit_v2_b200.lp import LP, Csr  # noqa: E402


def few_rows(n, k, rows, density, seed):
    """Portfolio-like QP with several rows: the budget and sparse ones."""
    rng = np.random.default_rng(seed)
    q = W.portfolio_qp(n, k, seed=seed)
    idx, ptr, val = [np.arange(n)], [0, n], [np.ones(n)]
    for r in range(1, rows):
        pick = np.flatnonzero(rng.random(n) < density / r)
        idx.append(pick)
        val.append(rng.uniform(0.5, 1.5, size=len(pick)))
        ptr.append(ptr[-1] + len(pick))
    A = Csr(rows, n, np.array(ptr), np.concatenate(idx), np.concatenate(val))
    lo = np.concatenate([[1.0], np.zeros(rows - 1)])
    hi = np.concatenate([[1.0], np.full(rows - 1, 0.9)])
    return LP(A, q.c, q.l, q.u, lo, hi, F=q.F, D=q.D)


def cases():
    # fewer columns than slices, one column a slice, remainders, the FP64 edge of
    # shared memory (100,000 x 50 has rows of F in L2), rank edges
    for n, k in ((5, 2), (592, 3), (1999, 1), (2050, 33), (20011, 64), (3001, 128), (70001, 50), (100_000, 50)):
        yield f"budget_{n}_{k}", W.portfolio_qp(n, k, seed=n)
    yield "two_rows", few_rows(9001, 20, 2, 0.5, 1)
    yield "four_rows", few_rows(700, 17, 4, 0.6, 2)
    yield "four_rows_long", few_rows(30_011, 9, 4, 0.3, 3)


def main(out):
    got = {}
    for name, lp in cases():
        for prec in ("Mixed", "Double", "Dynamic"):
            for ce, it in ((64, 128), (5, 15)):
                r = gb.solve_pdhg_gpu(lp, gb.Options(tol=1e-13, max_iter=it, check_every=ce,
                                                     precision=gb.Precision[prec]))
                got[f"{name}.{prec}.{ce}"] = np.concatenate([[r.iterations], r.x, r.y])
    np.savez(out, **got)


if __name__ == "__main__":
    main(sys.argv[1])
