"""A launch names no kernel but its own: CUDA loads each kernel when it is first
named, so a loop over every instantiation would load them all in a process's
first launch."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h261enc_cuda_b200", "csrc",
                      "kernels.cu")


def test_attributes_are_set_for_the_launched_kernel_only():
    text = re.sub(r"/\*.*?\*/", "", open(SOURCE).read(), flags=re.S)
    named = re.findall(r"cudaFunc\w+\(\s*([^;]*?),", text) + re.findall(r"cudaOccupancy\w+\(\s*&?\w+,\s*([^,]*),", text)
    assert named and all(n.strip() == "fn" for n in named), named
