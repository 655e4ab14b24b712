"""CPU: the reference arm of the benchmark script on a checkout without the
reference's compiled kernels says so and ends normally."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_its_kernels():
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "satan_ref_o3")):
        pytest.skip("the reference's kernels are built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "1"],
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout.splitlines()[-1])
    assert out["impl"] == "reference" and "satan_ref_o3" in out["unavailable"]
