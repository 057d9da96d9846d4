"""CPU suite: the benchmark's reference arm where the reference cannot be run."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("workload", ["c1_csr_add", "c4b_spgemm_laplacian"])
def test_reference_arm_without_the_reference(workload):
    """The arm times the reference or says that it cannot: it never times the oracle in its place."""
    from oracle.cpu_oracle import Reference
    if Reference.available() and "spgemm" not in workload:
        pytest.skip("the reference's kernels are built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--workload", workload, "--steps", "1", "--warmup", "3"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    line = json.loads(r.stdout)
    assert r.returncode == 0 and line["impl"] == "reference" and line["unavailable"] and "value" not in line
