"""bench.py's reference arm on a box to which the reference's sources never came: one line that says so, and success."""
import json
import os
import subprocess
import sys

import pytest

from oracle_lib import ref_available

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(ref_available("fp32") or ref_available("q8"), reason="the reference is there")
@pytest.mark.parametrize("quant", ["f32", "q8"])
def test_reference_arm_without_the_reference(quant):
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--quant", quant, "--steps", "2", "--warmup", "1"], capture_output=True, text=True,
                       timeout=120)
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert r.returncode == 0 and line["impl"] == "reference" and "not built" in line["unavailable"]
