"""bench.py --impl reference times the reference's own code or nothing: without a build of it, it says so in one line."""
import json
import os
import subprocess
import sys

import pytest

import oracle_lib as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unavailable_without_the_reference():
    if os.path.exists(O.REF_SO) or os.path.isdir(os.path.join(O.REF_TREE, "MDLIB")):
        pytest.skip("the reference is here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--size", "65", "--steps", "1", "--warmup", "1"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
