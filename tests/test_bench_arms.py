"""bench.py's arms, as far as they need no GPU."""
import json
import os
import subprocess
import sys

import pytest

from oracle import native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(impl):
    cmd = [sys.executable, os.path.join(ROOT, "bench.py"), "--impl", impl, "--steps", "1", "--warmup", "0",
           "--model", "llama-tiny", "--cpu-sample-mb", "1", "--no-cache"]
    done = subprocess.run(cmd, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert done.returncode == 0, done.stderr[-800:]
    return json.loads(done.stdout.strip().splitlines()[-1])


@pytest.mark.skipif(native.ref() is not None, reason="the reference's core is installed")
def test_no_stand_in_for_the_reference():
    line = _run("reference")
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_the_cpu_baseline_says_what_it_ran():
    line = _run("cpu")
    assert line["impl"] == "cpu" and line["cpu_baseline"]["value"] > 0
    assert line["cpu_baseline"]["kind"] == ("port" if native.ref() is None else "reference")
