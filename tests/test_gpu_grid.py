"""LPs kept by the whole GPU (k_grid) against the streaming kernels
(GANIT_B200_RESIDENT=0): FP32 and BF16 phases give the same bits; FP64 sums are
taken in another order: 64 iterations, rows of up to 1,024 entries, 8 for the
step sizes' weighting: 64 * 1030 * 8 * 1.1e-16 = 6e-11."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WORKER = os.path.join(os.path.dirname(__file__), "grid_worker.py")


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for on in ("1", "0"):
        f = str(tmp_path_factory.mktemp("grid") / f"r{on}.npz")
        p = subprocess.run([sys.executable, WORKER, f], env=dict(os.environ, GANIT_B200_RESIDENT=on, GANIT_B200_TRACE="1"),
                           capture_output=True, text=True, timeout=900)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append((dict(np.load(f)), p.stderr))
    return out


def test_both_precisions_ran_on_chip(both):
    assert "grid f32" in both[0][1] and "grid f64" in both[0][1]
    assert "grid f" not in both[1][1]


@pytest.mark.parametrize("prec", ["Mixed", "MixedBf16", "Double", "Dynamic"])
def test_on_chip_iterations_match_streamed_ones(both, prec):
    on, off = both[0][0], both[1][0]
    keys = [k for k in on if k.split(".")[1] == prec]
    assert len(keys) == 12 and set(on) == set(off)
    for k in keys:
        if prec in ("Mixed", "MixedBf16"):
            np.testing.assert_array_equal(on[k], off[k], err_msg=k)
        else:
            assert np.linalg.norm(on[k] - off[k]) <= 6e-11 * np.linalg.norm(off[k]), k
