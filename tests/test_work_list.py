"""The engine's kept work lists do not outlive the arena that holds them
(tests/work_list_check.cpp: the engine's host code built with g++ on a stand-in
for the CUDA runtime, in which an arena gets an earlier one's addresses)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="needs g++, CUDA's headers")
def test_work_list_after_the_arena_grew(tmp_path):
    exe = tmp_path / "work_list_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CUDA_INCLUDE, "-I",
                    os.path.join(ROOT, "h261enc_cuda_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "work_list_check.cpp"), "-ldl"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"
