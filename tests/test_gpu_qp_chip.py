"""QP iterations in one cooperative launch (k_qp_chip) against the streaming
kernels (GANIT_B200_RESIDENT=0): FP32 phases give the same bits; FP64 sums are
taken in another order: 128 iterations of sums over n <= 100,000 columns, each
within n 2^-53 relative, and PDHG's step does not expand differences:
128 * 100,000 * 1.1e-16 = 1.4e-9."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WORKER = os.path.join(os.path.dirname(__file__), "qp_chip_worker.py")


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for on in ("1", "0"):
        f = str(tmp_path_factory.mktemp("qp") / f"r{on}.npz")
        p = subprocess.run([sys.executable, WORKER, f], env=dict(os.environ, GANIT_B200_RESIDENT=on),
                           capture_output=True, text=True, timeout=900)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append(dict(np.load(f)))
    return out


@pytest.mark.parametrize("prec", ["Mixed", "Double", "Dynamic"])
def test_on_chip_qp_matches_streamed(both, prec):
    on, off = both
    keys = [k for k in on if k.split(".")[1] == prec]
    assert len(keys) == 22 and set(on) == set(off)
    for k in keys:
        if prec == "Mixed":
            np.testing.assert_array_equal(on[k], off[k], err_msg=k)
        else:
            assert np.linalg.norm(on[k] - off[k]) <= 1.4e-9 * np.linalg.norm(off[k]), k
