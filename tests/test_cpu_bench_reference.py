"""The benchmark's reference arm runs the reference's own program or says that it is unavailable: a
figure of this repository's restatement of it is no reference figure."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_is_the_reference_or_unavailable():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--res", "128", "--steps", "1"],
                         cwd=ROOT, capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference"
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "ref_cpu_dc")):
        assert line["cpu_baseline"]["kind"] == "reference" and line["value"] > 0
    else:
        assert line["unavailable"] and "value" not in line
