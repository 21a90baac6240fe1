"""The benchmark's reference arm where the compiled reference is absent: it says
so at once, for every workload, and prints no rate of a stand-in."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("workload", ["clustered", "plummer", "ensemble", "serve"])
def test_reference_arm_without_the_compiled_reference(workload):
    import ref_runner
    if ref_runner.available():
        pytest.skip("the compiled reference is here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--workload", workload, "--steps", "1"],
                       cwd=ROOT, stdout=subprocess.PIPE, timeout=120)
    assert r.returncode == 0
    out = json.loads(r.stdout.decode().strip().splitlines()[-1])
    assert out["impl"] == "reference" and out["unavailable"] and "value" not in out
