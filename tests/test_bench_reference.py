"""``bench.py --impl reference`` times the reference's own code or nothing: without
a build of it the line says so, and no code of this repository stands in."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference_says_unavailable():
    from oracle import oracle as O

    if O.ref_available():
        pytest.skip("the reference is built here: the arm would time it")
    p = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "2",
                        "--warmup", "1"], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert p.returncode == 0, p.stderr[-2000:]
    line = json.loads(p.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
