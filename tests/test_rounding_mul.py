"""The encode kernel's transforms multiply by the reference's double constants
and round the inverse DCT's output in float (mul_hilo and idct_round in
h261enc_cuda_b200/csrc/kernels.cu).  That is bit-exact only because the float
forms equal the double ones for every float that reaches them;
tests/rounding_check_mul.c checks them all (a few seconds)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_float_forms_equal_the_double_ones(tmp_path):
    exe = tmp_path / "rounding_check_mul"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fno-fast-math", "-o", str(exe),
                    os.path.join(ROOT, "tests", "rounding_check_mul.c"), "-lm"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    checked, differing = out.stdout.split()
    assert out.returncode == 0 and int(differing) == 0, f"{differing} floats differ"
    assert int(checked) > 700_000_000
