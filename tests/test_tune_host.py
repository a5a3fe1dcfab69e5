"""Builds and runs tests/cpp/test_tune.cpp on the CPU: which launch
configurations the autotuner may choose from."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tune_configurations(tmp_path):
    exe = str(tmp_path / "test_tune")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror",
                           "-I", os.path.join(ROOT, "tensor_train_gb300", "csrc"),
                           "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "test_tune.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
