"""The bench's reference arm runs the unmodified crate or says why not."""
import json
import subprocess
import sys
from pathlib import Path


def test_reference_arm_is_the_crate_or_nothing():
    root = Path(__file__).resolve().parent.parent
    for workload in ("large8192", "mesh96", "deformation512"):
        r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "3",
                            "--workload", workload], cwd=root, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        line = json.loads(r.stdout)
        assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
