"""Builds and runs tests/cpp/test_inner_sizes.cpp on the CPU: the buffers of an
inner-product chain."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_inner_sizes(tmp_path):
    exe = str(tmp_path / "test_inner_sizes")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror",
                           "-I", os.path.join(ROOT, "tensor_train_gb300", "csrc"),
                           "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "test_inner_sizes.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
