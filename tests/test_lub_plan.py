"""CPU test of the launch shapes of the blocked FP64 LU kernel."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_lub_plan_invariants(tmp_path):
    """bcr_lub_plan.cuh for every accepted shape: shared memory, threads per row, and
    never more CTAs than slabs, whatever the device answers about residency."""
    src = os.path.join(ROOT, "tests", "cpp", "lub_plan_check.cu")
    exe = str(tmp_path / "lub_plan_check")
    subprocess.run(["nvcc", "-std=c++17", "-cudart", "shared", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(ROOT, "alglin_b200", "csrc"), src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "0 failures" in r.stdout
