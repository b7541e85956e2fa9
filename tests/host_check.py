"""Builds and runs the checks of the core's host code (tests/*_check.cpp, on
the stand-in for the CUDA runtime in tests/fake_cuda.h)."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
AVAILABLE = shutil.which("g++") is not None and os.path.isdir(CUDA_INCLUDE)


def run(tmp_path, name, *args):
    exe = tmp_path / name
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CUDA_INCLUDE, "-I",
                    os.path.join(ROOT, "h261enc_cuda_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", name + ".cpp"), "-ldl"], check=True)
    out = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"
