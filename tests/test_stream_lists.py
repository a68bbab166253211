"""Row-block lists of the instances that stream while others of their batch
iterate on chip, host logic, no GPU: tests/stream_lists_check.cu builds them at
every level from schedules that differ by matrix type, as after autotuning,
and checks that each block indexes the bitmaps and slots of its own schedule."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_streamed_blocks_come_from_the_schedule_of_their_matrix_type(tmp_path):
    from ganit_v2_b200 import build

    exe = tmp_path / "stream_lists_check"
    cmd = [build.nvcc(), "-std=c++17", "-O1", *build.ARCH, "-o", str(exe), os.path.join(HERE, "stream_lists_check.cu"),
           os.path.join(build.CSRC, "gb_pool.cu")]
    out = subprocess.run(cmd, capture_output=True, text=True)
    if out.returncode != 0:
        pytest.fail("stream_lists_check.cu did not compile:\n" + out.stdout + out.stderr)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
    lines = run.stdout.strip().splitlines()
    assert len(lines) == 6 and all(line.startswith("ok ") for line in lines), run.stdout
