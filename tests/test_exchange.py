"""The exchange between the CTAs of a cluster when some own no rows or no
columns, host logic, no GPU: tests/exchange_check.cu runs a model of its
barriers on dealt shares with random delays and checks that no share of one
iteration lands in the phase of another."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_share_overtakes_another(tmp_path):
    from ganit_v2_b200 import build

    exe = tmp_path / "exchange_check"
    cmd = [build.nvcc(), "-std=c++17", "-O2", *build.ARCH, "-o", str(exe), os.path.join(HERE, "exchange_check.cu"),
           os.path.join(build.CSRC, "gb_pool.cu")]
    out = subprocess.run(cmd, capture_output=True, text=True)
    if out.returncode != 0:
        pytest.fail("exchange_check.cu did not compile:\n" + out.stdout + out.stderr)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
    lines = run.stdout.strip().splitlines()
    assert len(lines) == 6 and all(line.startswith("ok ") for line in lines), run.stdout
