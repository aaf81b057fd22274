"""The reference arm runs none of this repository's code: the reference cannot be
built here, and it says so."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_reference_arm():
    run = lambda rank: subprocess.run(  # noqa: E731
        [sys.executable, "bench.py", "--impl", "reference", "--gpus", "2", "--steps", "1", "--warmup", "0"], cwd=ROOT,
        env={**os.environ, "RANK": rank}, check=True, capture_output=True, text=True).stdout
    line = json.loads(run("0"))
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
    assert run("1") == ""
