"""CPU: `bench.py --impl reference` times the reference's own compiled kernels or says that they are unavailable - never
this repository's oracle."""
import json
import os
import subprocess
import sys

from conftest import ROOT
from oracle.inkq_oracle import Reference


def test_reference_arm_runs_the_reference_or_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "1", "--min-seconds", "0"],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference"
    if Reference.available_path()[0] is None:
        assert set(line) == {"impl", "unavailable"} and line["unavailable"]
    else:
        assert line["cpu_baseline"]["kind"] == "reference" and line["value"] > 0
