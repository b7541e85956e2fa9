"""Both sides of the limit up to which a step's descriptors and pictures go to
the device by a kernel (H261B_FETCH_MAX): below it that kernel also clears the
squared-error sums, above it the copy engine moves the bytes and a separate
clear precedes them.  With PSNR, with and without levels, with and without
sessions that write no bitstream, launched directly and replayed as graphs,
each side gives the oracle's bytes, reconstructions and squared errors.  The
side is read off the bytes that the step reports.  Integers: equality."""
import functools
import os
import re

import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu
HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h261enc_cuda_b200", "csrc",
                      "h261b_device.h")
W, H, N, QUANT = 352, 288, 3, 9
PICTURE = W * H * 3 // 2


def _limit():
    a, b = re.search(r"#define H261B_FETCH_MAX \((\d+) \* (\d+)\)", open(HEADER).read()).groups()
    return int(a) * int(b)


@functools.lru_cache(maxsize=None)
def _stream(k):
    clip = synth.clip(2, W, H, 900 + k, N)
    return clip, O.encode_stream(clip, W, H, quant=QUANT)


@pytest.mark.parametrize("above", [0, 1])
@pytest.mark.parametrize("plain", [0, 1])
@pytest.mark.parametrize("levels", [0, 1])
@pytest.mark.parametrize("graphs", [0, 1])
def test_both_sides_of_the_limit(gpu, above, plain, levels, graphs):
    """`plain` of the sessions write no bitstream."""
    # the most CIF pictures whose bytes and descriptors (some 2 KB each) fit, or one more
    n = _limit() // (PICTURE + 2048) + above
    streams = [_stream(k) for k in range(n)]
    with Engine(levels_to_host=levels, use_graphs=graphs, warps_per_cta=8, kernel_split=1, tail_items=1,
                staging=1) as e:
        for turn in range(4):
            # each clip four times over, as new sessions: steps of one signature, which replay as graphs
            sids = [e.open(W, H, QUANT, bitstream=int(k >= plain), psnr=1) for k in range(n)]
            off = [0] * n
            for i in range(N):
                e.submit_frames(sids, [clip[i] for clip, _ in streams])
                e.step()
                e.sync()
                up = e.last_copy_bytes()[0]
                assert n * PICTURE < up and (up > _limit()) == bool(above), up
                for k, sid in enumerate(sids):
                    clip, (bits, sizes, _, recon) = streams[k]
                    r = e.result(sid)
                    planes = np.concatenate(e.recon(sid))
                    assert np.array_equal(planes, recon[i]), f"session {k} picture {i}: reconstruction"
                    d = clip[i].astype(np.int64) - planes
                    assert r.ssd == tuple(int((p * p).sum()) for p in synth.split(d, W, H)), f"session {k} picture {i}"
                    assert (r.levels is not None) == bool(levels)
                    if k >= plain:
                        assert r.bits == bits[off[k]:off[k] + sizes[i]], f"session {k} picture {i}: bytes"
                        off[k] += sizes[i]
                    else:
                        assert r.bits is None
            for sid in sids:
                e.close(sid)
        if graphs:
            assert e.graph_stats()[1] > 0
