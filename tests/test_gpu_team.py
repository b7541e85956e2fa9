"""Small launches take a CTA of four warps per macroblock (at most four
macroblocks a multiprocessor: 592), larger ones a warp each; a configured
launch shape keeps the warp.  Both, through the engine and through the
no-allocation entry point, give the oracle's records, levels and
reconstructions, with both searches, both arithmetics, and an intra refresh.
Integers: equality."""
import ctypes

import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine
from test_zz_no_alloc import DevPicture, NoallocPicture, _lib_noalloc, _lib_state_bytes

pytestmark = pytest.mark.gpu
N, QUANT = 4, 6
# one MB; an odd grid; the last size with a team per MB (592 MBs); the first without
SIZES = [(16, 16), (80, 48), (592, 256), (608, 256)]


def _clip(w, h):
    big = synth.clip(3, max(w, 64), max(h, 64), w + h, N)
    if w >= 64 and h >= 64:
        return big
    cut = [np.concatenate([p.reshape(-1, max(w, 64) // k)[:h // k, :w // k].ravel()
                           for p, k in zip(synth.split(f, max(w, 64), max(h, 64)), (1, 2, 2))]) for f in big]
    return np.stack(cut)


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("me_mode,fmad", [(0, 1), (1, 0)])
def test_sizes_around_the_line(gpu, w, h, me_mode, fmad):
    import torch
    frames = _clip(w, h)
    want = O.encode_sequence(frames, w, h, QUANT, me_mode=me_mode, fmad=fmad)
    for shape in (0, 4):
        with Engine(me_mode=me_mode, fmad=fmad, warps_per_cta=shape) as e:
            sid = e.open(w, h, QUANT)
            for i in range(N):
                e.submit_frame(sid, frames[i])
                e.step()
                e.sync()
                assert np.array_equal(e.result(sid).to_abi(w)["tcoeff"], want["mbs"][i]["tcoeff"]), (shape, i)
                assert np.array_equal(e.result(sid).to_abi(w)["mv"], want["mbs"][i]["mv"]), (shape, i)
                assert np.array_equal(np.concatenate(e.recon(sid)), want["recon"][i]), (shape, i)
    lib = _lib_noalloc()
    nmb = (w // 16) * (h // 16)
    cur = [DevPicture(torch, w, h, frames[i]) for i in range(N)]
    rec = [DevPicture(torch, w, h) for _ in range(2)]
    state = torch.zeros(_lib_state_bytes(), dtype=torch.uint8, device="cuda:0")
    mbs = torch.zeros(nmb * 16, dtype=torch.uint8, device="cuda:0")
    levels = torch.zeros(nmb * 384, dtype=torch.int8, device="cuda:0")
    torch.cuda.synchronize()
    for i in range(N):
        p = NoallocPicture(w, h, int(i > 0), QUANT, me_mode, fmad, 5, int(i == 0), *cur[i].planes(),
                           *rec[(i + 1) & 1].planes(), *rec[i & 1].planes(), state.data_ptr(), mbs.data_ptr(),
                           levels.data_ptr())
        assert lib.h261b_encode_picture_noalloc(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert np.array_equal(rec[i & 1].host(), want["recon"][i]), f"no-allocation picture {i}"


@pytest.mark.parametrize("quant,bitrate", [(0, 96000), (9, 0)])
def test_bitstream_rate_control_and_errors(gpu, quant, bitrate):
    w, h, n = 176, 144, 8
    frames = synth.clip(2, w, h, 77, n)
    bits, nb, nq, recon = O.encode_stream(frames, w, h, quant=quant, bitrate=bitrate or 384000, intra_period=3)
    got = {}
    for shape in (0, 8):
        with Engine(levels_to_host=shape // 8, warps_per_cta=shape) as e:
            sid = e.open(w, h, quant or 10, intra_period=3, bitstream=1, rate_control=int(not quant),
                         bitrate=bitrate, psnr=1)
            out, off = [], 0
            for i in range(n):
                e.submit_frame(sid, frames[i])
                e.step()
                e.sync()
                r = e.result(sid)
                assert r.bits == bits[off:off + nb[i]] and r.quant == nq[i], (shape, i)
                assert np.array_equal(np.concatenate(e.recon(sid)), recon[i]), (shape, i)
                off += nb[i]
                out.append((r.mbs.tobytes(), r.ssd))
            got[shape] = out
    assert got[0] == got[8]
