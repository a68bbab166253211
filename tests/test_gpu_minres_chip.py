"""The differentiable layer's MINRES on chip (k_mr_solve_chip) at the sizes
where its form changes: one row per thread (up to 512 free columns and active
rows), two (up to 1,024), and beyond, where k_mr_solve takes over; uneven
instances share a launch.  Against the dense basis sensitivities: a relative
residual of 1e-10 and a basis condition of at most 5e4 bound the error by
5e-6."""
import numpy as np
import pytest

from ganit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(3, 7, 2)], [(40, 90, 5), (60, 130, 6)], [(520, 1100, 10), (30, 61, 4)],
                                    [(600, 1300, 8), (200, 420, 10)], [(1250, 2600, 14)]])
def test_gradients_match_basis_sensitivities(shapes):
    import ganit_v2_b200 as gb

    lps = [W.nondegenerate_lp(m, n, k, seed=9000 + i, max_cond=5e4) for i, (m, n, k) in enumerate(shapes)]
    opt = gb.Options(tol=1e-6, precision=gb.Precision.Mixed)
    ds = gb.DiffSolver(lps, opt, tail_iters=40, ckpt_every=10)
    _, x, y = ds.forward(opt)
    rng = np.random.default_rng(1)
    w, v = rng.standard_normal(int(ds.n_off[-1])), rng.standard_normal(int(ds.m_off[-1]))
    g = ds.backward(w, v)
    for i, lp in enumerate(lps):
        n0, m0 = int(ds.n_off[i]), int(ds.m_off[i])
        f, d = lp.meta["interior"], lp.meta["tight"]
        assert ds.info(i)["polished"] and ds.info(i)["implicit_converged"]
        B = lp.A.to_scipy().tocsr()[np.flatnonzero(d)][:, np.flatnonzero(f)].toarray()
        q, p = np.zeros(lp.n), np.zeros(lp.m)
        q[f] = np.linalg.solve(B, v[m0:m0 + lp.m][d])
        p[d] = np.linalg.solve(B.T, w[n0:n0 + lp.n][f])
        for got, want in ((x[n0:n0 + lp.n], lp.meta["x0"]), (y[m0:m0 + lp.m], lp.meta["y0"]),
                          (g["c"][n0:n0 + lp.n], q), ((g["lo"] + g["hi"])[m0:m0 + lp.m], p)):
            assert np.linalg.norm(got - want) <= 5e-6 * np.linalg.norm(want)
    ds.close()
