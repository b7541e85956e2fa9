"""After its first call on a device, h261b_encode_picture_noalloc can be
captured into a CUDA graph whatever the picture's size, search and arithmetic
are, also where the capture is the first call with them: no kernel is left to
be set up then.  The replayed graphs give the oracle's reconstructions.
In a process of its own, in which nothing has run before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, sys
sys.path[:0] = [ROOT, ROOT + "/oracle", ROOT + "/tests"]
import numpy as np
import torch
import oracle as O
from h261enc_cuda_b200 import synth
from test_zz_no_alloc import DevPicture, NoallocPicture, _lib_noalloc, _lib_state_bytes

lib = _lib_noalloc()
N, QUANT = 3, 7


class Stream:
    def __init__(self, w, h, me_mode, fmad):
        self.frames = synth.clip(2, w, h, 60 + w + me_mode, N)
        self.want = O.encode_sequence(self.frames, w, h, QUANT, me_mode=me_mode, fmad=fmad)["recon"]
        self.cur = [DevPicture(torch, w, h, f) for f in self.frames]
        self.rec = [DevPicture(torch, w, h) for _ in range(N + 1)]
        nmb = w * h // 256
        self.keep = [torch.zeros(n, dtype=torch.uint8, device="cuda:0") for n in (_lib_state_bytes(), 16 * nmb, 384 * nmb)]
        self.pics = [NoallocPicture(w, h, int(i > 0), QUANT, me_mode, fmad, 5, int(i == 0), *self.cur[i].planes(),
                                    *self.rec[i].planes(), *self.rec[i + 1].planes(),
                                    *(k.data_ptr() for k in self.keep)) for i in range(N)]

    def encode(self):
        for p in self.pics:
            rc = lib.h261b_encode_picture_noalloc(ctypes.byref(p), torch.cuda.current_stream().cuda_stream)
            assert rc == 0, lib.h261b_last_error()

    def check(self):
        for i in range(N):
            assert np.array_equal(self.rec[i + 1].host(), self.want[i]), i


first = Stream(64, 64, 0, 1)
rest = [Stream(w, h, me_mode, fmad) for w, h in ((176, 144), (640, 256)) for me_mode in (0, 1) for fmad in (1, 0)]
first.encode()
torch.cuda.synchronize()
first.check()
for s in rest:
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=MODE):
        s.encode()
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        s.check()
print("ok")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_first_use_inside_a_capture(gpu, mode):
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nMODE = {mode!r}\n" + CHILD], capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
