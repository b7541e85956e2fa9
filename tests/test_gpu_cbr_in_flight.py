"""The QUANT reported with a rate-controlled picture is the one its bytes were
coded with, with three steps in flight: the rate control of the next step
chooses the next picture's QUANT as soon as this picture is laid out, while
its bytes are still being packed.  So nothing after the layout may read the
rate control's live state.  Integers: equality with the oracle's frame loop."""
import os
import re

import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h261enc_cuda_b200", "csrc",
                      "bitstream.cu")


def test_nothing_after_the_layout_reads_the_rate_control():
    text = open(SOURCE).read()
    after = re.sub(r"/\*.*?\*/", "", text[text.index("constexpr int PACK_DONE_MAX"):text.index("} // namespace\n} //")],
                   flags=re.S)
    assert "copy_picture(" in after and "pack_kernel(" in after
    assert not re.search(r"\brc\b", after)


@pytest.mark.gpu
@pytest.mark.parametrize("sessions", [1, 4])
@pytest.mark.parametrize("graphs", [0, 1])
def test_quant_of_pictures_in_flight(gpu, sessions, graphs):
    w, h, n = 176, 144, 48
    rates = [96000, 64000, 160000, 320000][:sessions]
    clips = [synth.clip(3, w, h, 300 + k, n) for k in range(sessions)]
    want = [O.encode_stream(c, w, h, quant=0, bitrate=b) for c, b in zip(clips, rates)]
    assert all(len(set(x[2])) > 2 for x in want)   # a QUANT that changes
    quants, got = [[] for _ in rates], [b"" for _ in rates]
    with Engine(levels_to_host=0, use_graphs=graphs) as e:
        sids = [e.open(w, h, 10, bitstream=1, rate_control=1, bitrate=b) for b in rates]

        def read(k):
            e.wait_step(k)
            for j, sid in enumerate(sids):
                r = e.result(sid)
                assert r.frame_index == k
                quants[j].append(r.quant)
                got[j] += r.bits

        for k in range(n):
            e.submit_frames(sids, [c[k] for c in clips])
            e.step()
            if k >= 2:
                read(k - 2)
        read(n - 2)
        read(n - 1)
    for j in range(sessions):
        assert quants[j] == list(want[j][2]), f"session {j}"
        assert got[j] == want[j][0], f"session {j}: bytes"
