"""Objects that the coding kernels read and write as 16-byte words are aligned
to 16 bytes by their types, in device, shared and constant memory alike, and
not only by what lies before them.  Compiled with nvcc; nothing runs."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h261enc_cuda_b200", "csrc")

CHECK = """
#include <cuda_runtime.h>
#include "vlc_coder.h"
using namespace h261b;
struct Holder { char first; VlcTables tables; VlcScratch scratch; };   /* after an odd member */
static_assert(alignof(VlcTables) >= 16 && sizeof(VlcTables) % 16 == 0, "code tables");
static_assert(alignof(VlcScratch) >= 16, "coder's memory");
static_assert(offsetof(Holder, tables) % 16 == 0 && offsetof(Holder, scratch) % 16 == 0, "members");
static_assert(offsetof(VlcTables, cm) % 4 == 0, "zig-zag order, read as 4-byte words");
static_assert(offsetof(VlcScratch, cm) % 8 == 0 && offsetof(VlcScratch, level) % 4 == 0, "levels");
static_assert(offsetof(h261b_denoise_dev_t, offset) % 16 == 0, "denoise offsets, a column a load");
static_assert(sizeof(h261b_mb_info_t) == 16, "records, one a load");
static_assert(sizeof(h261b_session_dev_t) % 8 == 0 && sizeof(h261b_step_dev_t) % 256 == 0, "descriptors");
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_wide_access_is_aligned_by_type(tmp_path):
    src = tmp_path / "alignment.cu"
    src.write_text(CHECK)
    out = subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, "-c", "-o",
                          str(tmp_path / "alignment.o"), str(src)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
