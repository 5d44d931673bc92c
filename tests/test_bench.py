"""bench.py's reference arm without GALIC's own C, on the CPU."""
import json
import os
import subprocess
import sys

import pytest

import oracle_lib
from conftest import ROOT


@pytest.mark.skipif(oracle_lib.reference_available(), reason="GALIC's own C (oracle/_ref) is built")
def test_reference_arm_names_no_baseline_that_it_did_not_run():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup",
                          "0", "--cpu-seconds", "1", "--scale", "0.001"], cwd=ROOT, check=True, capture_output=True,
                         text=True, timeout=300).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
