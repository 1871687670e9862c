"""bench.py --impl reference: the reference's own objects, or the statement that they are not there."""
import json
import subprocess
import sys
from pathlib import Path

import pytest


def test_nothing_else_is_timed_under_the_reference_s_name():
    import oracle
    if oracle.reference_available():
        pytest.skip("the reference's objects are built here")
    root = Path(__file__).resolve().parent.parent
    done = subprocess.run([sys.executable, str(root / "bench.py"), "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "3"],
                          capture_output=True, text=True, timeout=300, cwd=root)
    assert done.returncode == 0, done.stderr
    line = json.loads(done.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
