"""On-chip iterations of small instances, host logic, no GPU:
tests/resident_check.cu deals instances to clusters of every size and follows
the packing arithmetic (positions and packed entries written once, inside
their CTA's share; slice sums bit for bit the streaming kernels' FP32 sums)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_resident_plan_and_packing(tmp_path):
    from ganit_v2_b200 import build

    exe = tmp_path / "resident_check"
    cmd = [build.nvcc(), "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", *build.ARCH, "-o", str(exe),
           os.path.join(HERE, "resident_check.cu"), os.path.join(build.CSRC, "gb_pool.cu")]
    out = subprocess.run(cmd, capture_output=True, text=True)
    if out.returncode != 0:
        pytest.fail("resident_check.cu did not compile:\n" + out.stdout + out.stderr)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
    lines = run.stdout.strip().splitlines()
    assert len(lines) == 50 and all(line.startswith("ok ") for line in lines), run.stdout
