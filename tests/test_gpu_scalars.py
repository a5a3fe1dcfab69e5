"""Builds and runs tests/cpp/test_scalars.cu: the FP64 scalars formed from the
hardware's approximations hold their stated bounds over FP64's range."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_scalars_over_the_range(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "test_scalars")
    subprocess.check_call([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-I", os.path.join(ROOT, "tensor_train_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "test_scalars.cu"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
