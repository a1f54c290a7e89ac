"""The benchmark's reference arm times the reference's own build or nothing: never this repository's restatement of it."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_is_the_reference_or_unavailable():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "3",
                          "--cpu-sample-rows", "2000"], stdout=subprocess.PIPE, text=True, timeout=300, check=True).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["impl"] == "reference"
    from oracle import ref_binding
    if ref_binding.available():
        assert line["cpu_baseline"]["kind"] != "port" and line["value"] > 0
    else:
        assert line["unavailable"] and "value" not in line
