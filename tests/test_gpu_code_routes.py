"""Macroblocks are coded to bit strings by the warp that encodes them in small
steps (at most 16 macroblocks a multiprocessor) and by the codes kernel in
larger ones.  On both sides of that line, with QUANT from 1 (escapes, blocks
full of levels) to 31 (few or none) and intra refresh, the bytes are the
oracle's."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu
W, H, N = 176, 144, 4
QUANTS = [1, 2, 3, 5, 8, 13, 21, 31]


# 99 macroblocks a picture: 23 pictures are 2,277 and 24 are 2,376, around 16 x 148
@pytest.mark.parametrize("sessions", [1, 23, 24])
@pytest.mark.parametrize("preset", [2, 3])
def test_both_sides_of_the_line(gpu, sessions, preset):
    clips = [synth.clip(preset, W, H, 700 + k % 8, N) for k in range(min(sessions, 8))]
    want = [O.encode_stream(c, W, H, quant=q, intra_period=3) for c, q in zip(clips, QUANTS)]
    with Engine(levels_to_host=0) as e:
        sids = [e.open(W, H, QUANTS[k % 8], intra_period=3, bitstream=1) for k in range(sessions)]
        at = [0] * sessions
        for i in range(N):
            e.submit_frames(sids, [clips[k % 8][i] for k in range(sessions)])
            e.step()
            e.sync()
            for k, sid in enumerate(sids):
                bits, sizes = want[k % 8][:2]
                assert e.result(sid).bits == bits[at[k]:at[k] + sizes[i]], f"session {k} picture {i}"
                at[k] += sizes[i]
