"""Small launches that take a team of four warps per macroblock, on inter
pictures: engines with open knobs whose launch-plan trial is over (the trial's
own steps take the warp-per-macroblock kernel), at the edges of the team's
range.  Records, levels, vectors, reconstructions and bytes are the oracle's,
with both searches and both arithmetics.  Integers: equality."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine
from test_gpu_team import SIZES, _clip

pytestmark = pytest.mark.gpu
N, QUANT = 4, 6


@pytest.fixture(scope="module")
def tuned(gpu):
    """A process whose trial is over: 27 steps of mostly inter pictures."""
    clip = synth.clip(2, 64, 64, 1, 8)
    with Engine() as e:
        sid = e.open(64, 64, QUANT)
        for i in range(40):
            if not e.plan()[0]["tuning"] and e.plan()[0]["source"]:
                return
            e.submit_frame(sid, clip[i % 8])
            e.step()
            e.sync()
    pytest.fail("the trial did not end")


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("me_mode,fmad", [(0, 1), (1, 1), (0, 0)])
def test_inter_pictures_at_the_edges(gpu, tuned, w, h, me_mode, fmad):
    frames = _clip(w, h)
    want = O.encode_sequence(frames, w, h, QUANT, me_mode=me_mode, fmad=fmad)
    with Engine(me_mode=me_mode, fmad=fmad) as e:
        assert e.plan()[0]["source"] == 2 and not e.plan()[0]["tuning"]
        sid = e.open(w, h, QUANT)
        for i in range(N):
            e.submit_frame(sid, frames[i])
            e.step()
            e.sync()
            got, exp = e.result(sid).to_abi(w), want["mbs"][i]
            for f in ("type", "flags", "quant", "cbp", "mv", "tcoeff"):
                assert np.array_equal(got[f], exp[f]), (i, f)
            assert np.array_equal(np.concatenate(e.recon(sid)), want["recon"][i]), i


@pytest.mark.parametrize("quant,bitrate", [(0, 96000), (9, 0)])
@pytest.mark.parametrize("levels", [0, 1])
def test_bitstream_of_inter_pictures(gpu, tuned, quant, bitrate, levels):
    w, h, n = 176, 144, 10
    frames = synth.clip(2, w, h, 78, n)
    bits, nb, nq, recon = O.encode_stream(frames, w, h, quant=quant, bitrate=bitrate or 384000)
    with Engine(levels_to_host=levels) as e:
        assert e.plan()[0]["source"] == 2 and not e.plan()[0]["tuning"]
        sid = e.open(w, h, quant or 10, bitstream=1, rate_control=int(not quant), bitrate=bitrate, psnr=1)
        off = 0
        for i in range(n):
            e.submit_frame(sid, frames[i])
            e.step()
            e.sync()
            r = e.result(sid)
            planes = np.concatenate(e.recon(sid))
            assert r.bits == bits[off:off + nb[i]] and r.quant == nq[i], i
            assert np.array_equal(planes, recon[i]), i
            d = frames[i].astype(np.int64) - planes
            assert r.ssd == tuple(int((p * p).sum()) for p in synth.split(d, w, h)), i
            off += nb[i]
