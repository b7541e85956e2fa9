"""A process loads the kernels that it uses.  CUDA loads each kernel when it is
first named, and with the first one its whole module: so a launch names no
kernel but its own, and the encode kernels are eight modules (two arithmetics,
two searches, two staging variants)."""
import os
import re
import shutil
import subprocess

import pytest

from h261enc_cuda_b200 import _lib

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h261enc_cuda_b200", "csrc",
                      "launch.cu")


def test_attributes_are_set_for_the_launched_kernel_only():
    text = re.sub(r"/\*.*?\*/", "", open(SOURCE).read(), flags=re.S)
    named = re.findall(r"cudaFunc\w+\(\s*([^;]*?),", text) + re.findall(r"cudaOccupancy\w+\(\s*&?\w+,\s*([^,]*),", text)
    assert named and all(n.strip() == "fn" for n in named), named


@pytest.mark.skipif(shutil.which("readelf") is None, reason="needs readelf")
def test_encode_kernels_are_eight_modules():
    out = subprocess.run(["readelf", "-SW", _lib.core()._name], capture_output=True, text=True, check=True).stdout
    size = int(re.search(r"\.nvFatBinSegment\s+PROGBITS\s+\S+\s+\S+\s+(\S+)", out).group(1), 16)
    # a 24-byte entry per module: the eight, and those of the other sources
    assert size // 24 >= 8 + 5
