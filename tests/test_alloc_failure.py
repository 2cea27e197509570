"""A failed device allocation leaves the training step's buffers in a state that the next call repairs."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_train_buffers_after_a_failed_allocation(tmp_path):
    exe = str(tmp_path / "alloc_failure")
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "shared",
                    "-I", os.path.join(ROOT, "volumesurfacediscretemeshoptimization_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "test_alloc_failure.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
