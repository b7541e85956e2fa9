"""Steps whose sessions change from one to the next: other sizes in the same
number, the same sizes in another order, rate-controlled sessions among them,
a session closed with a picture queued and its slot opened again.  A step
writes its work list only when the sizes of its sessions differ from those of
the slot's last step; every session's bytes are the oracle's either way."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu
Q, C = (176, 144), (352, 288)
# (size, QUANT or 0 for CBR) of eight sessions
SESSIONS = [(Q, 8), (C, 12), (Q, 16), (C, 0), (Q, 0), (Q, 4), (C, 20), (Q, 8)]
# the sessions of each step, over three slots and more than one round of them
STEPS = [[0, 1], [0, 1], [0, 1], [0, 1], [0, 6], [2, 1], [0, 2], [1, 6], [0, 1, 3], [0, 3, 4], [5, 6, 4], [0, 1, 3],
         [0, 1, 3], [0, 1, 3], [0, 1, 3], [7], [5], [3], [1], [7, 5], [7, 5], [7, 5], [7, 5], [0, 1]]


@pytest.mark.parametrize("graphs", [0, 1])
def test_changing_sessions(gpu, graphs):
    n = len(STEPS)
    clips = [synth.clip(2, w, h, 900 + k, n) for k, ((w, h), _) in enumerate(SESSIONS)]
    want = [O.encode_stream(c, w, h, quant=q, bitrate=256000) for c, ((w, h), q) in zip(clips, SESSIONS)]
    with Engine(levels_to_host=0, use_graphs=graphs, max_sessions=16) as e:
        sids = [e.open(w, h, q, bitstream=1) if q else e.open(w, h, 10, bitstream=1, rate_control=1, bitrate=256000)
                for (w, h), q in SESSIONS]
        at, off = [0] * len(sids), [0] * len(sids)
        for t, step in enumerate(STEPS):
            # a session that goes before its picture is encoded, and the next one in its slot, which has none
            gone = e.open(*Q, 8, bitstream=1)
            e.submit_frame(gone, clips[0][0])
            e.close(gone)
            spare = e.open(*C, 8, bitstream=1)
            assert spare == gone
            for k in (step if t % 2 else step[::-1]):   # queued in any order
                e.submit_frame(sids[k], clips[k][at[k]])
            assert e.step() == len(step)
            e.sync()
            e.close(spare)
            pics, _ = e.step_pictures()
            assert list(pics["session_id"]) == sorted(sids[k] for k in step)
            for k in step:
                bits, sizes = want[k][:2]
                assert e.result(sids[k]).bits == bits[off[k]:off[k] + sizes[at[k]]], f"step {t} session {k}"
                off[k] += sizes[at[k]]
                at[k] += 1
        assert e.step() == 0   # nothing queued


def test_changing_sessions_do_not_capture_again(gpu):
    """Streams of a few pictures that end and begin keep the step's shape; their steps replay the slots' graphs (at
    most two a slot: with the work list's upload and without), as steps of unchanged sessions do."""
    rng = np.random.default_rng(5)
    clips = {s: synth.clip(2, *s, 77, 4) for s in (Q, C)}
    with Engine(max_sessions=16) as e:
        live = [(e.open(*s, 10, bitstream=1), s) for s in (Q, C, Q, Q, C, Q)]

        def steps(k, churn):
            for t in range(k):
                if churn and t % 4 == 0:
                    # a stream of each size ends and its successor begins, in the other's slot
                    for s in (Q, C):
                        i = int(rng.choice([j for j, (_, z) in enumerate(live) if z == s]))
                        e.close(live.pop(i)[0])
                    live.extend((e.open(*s, 10, bitstream=1), s) for s in ((C, Q) if rng.random() < 0.5 else (Q, C)))
                for sid, s in live:
                    e.submit_frame(sid, clips[s][t % 4])
                assert e.step() == len(live)
            e.sync()

        steps(60, False)      # the plan's trial, and the graphs of unchanged sessions
        before, _ = e.graph_stats()
        steps(120, True)
        captures, replays = e.graph_stats()
    assert captures - before <= 2 * 3
    assert replays >= 100
