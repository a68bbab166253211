"""Iterations of small instances on chip (k_resident) against the streaming
kernels (GANIT_B200_RESIDENT=0): the FP32 and BF16 phases give the same bits;
FP64 sums are taken in another order, so an iterate of K iterations may
differ by K (L + 6) 2^-53 relative per row of length L <= 1024 (PDHG's step
does not expand differences in its norm; 8 for the step sizes' weighting):
128 * 1030 * 8 * 1.1e-16 = 1.2e-10."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WORKER = os.path.join(os.path.dirname(__file__), "resident_worker.py")


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for on in ("1", "0"):
        f = str(tmp_path_factory.mktemp("res") / f"r{on}.npz")
        p = subprocess.run([sys.executable, WORKER, f], env=dict(os.environ, GANIT_B200_RESIDENT=on, GANIT_B200_TRACE="1"),
                           capture_output=True, text=True, timeout=900)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append((dict(np.load(f)), p.stderr))
    return out


def test_every_cluster_size_ran_on_chip(both):
    for c in (1, 2, 4, 8, 16):
        assert f"in clusters of {c}," in both[0][1], c
    assert "resident f" not in both[1][1]


@pytest.mark.parametrize("prec", ["Mixed", "MixedBf16", "Double", "Dynamic"])
def test_on_chip_iterations_match_streamed_ones(both, prec):
    on, off = both[0][0], both[1][0]
    keys = [k for k in on if not k.startswith("norm.") and k.split(".")[1] == prec]
    assert len(keys) > 40 and set(on) == set(off)
    for k in keys:
        if prec in ("Mixed", "MixedBf16"):
            np.testing.assert_array_equal(on[k], off[k], err_msg=k)
        else:
            assert np.linalg.norm(on[k] - off[k]) <= 1.2e-10 * np.linalg.norm(off[k]), k


def test_power_iteration_on_chip_gives_the_same_norm(both):
    """50 steps, each a sum over at most 1,024 entries of a row and one over
    7,501 columns: 50 * 8,525 * 1.1e-16 = 4.7e-11."""
    on, off = both[0][0], both[1][0]
    keys = [k for k in on if k.startswith("norm.")]
    assert len(keys) == 18
    for k in keys:
        assert abs(on[k] - off[k]) <= 4.7e-11 * off[k], k
