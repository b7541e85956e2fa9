"""The reference's sixteen device calls around the size up to which they take a
team of warps per macroblock (592), one encoder after another of another size,
planes uploaded twice before they are used and from memory that the caller
overwrites at once: motion estimation, levels and reconstructions are the
oracle's.  Integers: equality."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.compat import Boundary

pytestmark = pytest.mark.gpu
N, QUANT = 3, 9


@pytest.mark.parametrize("w,h", [(64, 64), (592, 256), (608, 256), (176, 144)])
def test_boundary(gpu, w, h):
    frames = synth.clip(3, w, h, w * 3 + h, N)
    want = O.encode_sequence(frames, w, h, QUANT)
    b = Boundary(w, h, denoise=5)
    try:
        ref = tuple(np.zeros_like(p) for p in synth.split(frames[0], w, h))
        for i in range(N):
            planes = [p.copy() for p in synth.split(frames[i], w, h)]
            noise = [np.full_like(p, 77) for p in planes]
            b.set_current(*noise)              # replaced before anything reads it
            b.set_current(*planes)
            b.set_reference(*noise)
            b.set_reference(*ref)
            for p in planes:
                p[:] = 0                       # the library has its own copy
            me = b.motion_estimation()
            if i:                              # the oracle searches no intra picture
                for f in ("intra", "cost", "fcost", "mvx", "mvy"):
                    assert np.array_equal(me[f], want["me"][i][f]), f"picture {i}: {f}"
            got = b.encode(want["md"][i], QUANT, int(i > 0))
            for f in ("type", "flags", "quant", "cbp", "mv", "tcoeff", "mb_x", "mb_y"):
                assert np.array_equal(got[f], want["mbs"][i][f]), f"picture {i}: {f}"
            ref = b.decode()
            assert np.array_equal(np.concatenate(ref), want["recon"][i]), f"picture {i}: reconstruction"
    finally:
        b.close()
