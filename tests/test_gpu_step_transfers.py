"""A step's transfers take the routes that its sizes and options choose: the
uploads of a small step (descriptors and pictures up to 256 KB) by a kernel, of
a larger one by the copy engine; the records and squared errors written to the
host by the pack kernel when every picture is a bitstream and no levels are
wanted, by a copy otherwise.  Each route gives the oracle's bytes,
reconstructions and squared errors; records agree with the bytes.  Integers
throughout: equality, no tolerance."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200 import synth
from h261enc_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu
W, H, N, QUANT = 176, 144, 4, 8


# six QCIF pictures and their descriptors stay below the limit, seven do not
@pytest.mark.parametrize("sessions", [1, 6, 7])
@pytest.mark.parametrize("plain,levels", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("graphs", [0, 1])
def test_every_route(gpu, sessions, plain, levels, graphs):
    """`plain` more sessions write no bitstream."""
    clips = [synth.clip(2, W, H, 500 + k, N) for k in range(sessions + plain)]
    want = [O.encode_stream(c, W, H, quant=QUANT) for c in clips]
    with Engine(levels_to_host=levels, use_graphs=graphs, warps_per_cta=8, kernel_split=1, tail_items=1,
                staging=1) as e:
        sids = [e.open(W, H, QUANT, bitstream=int(k < sessions), psnr=1) for k in range(sessions + plain)]
        off = [0] * len(sids)
        for i in range(3 * N):
            # each clip three times over, as new sessions, so that steps replay their graphs
            if i and i % N == 0:
                for sid in sids:
                    e.close(sid)
                sids = [e.open(W, H, QUANT, bitstream=int(k < sessions), psnr=1) for k in range(sessions + plain)]
                off = [0] * len(sids)
            e.submit_frames(sids, [c[i % N] for c in clips])
            e.step()
            e.sync()
            for k, sid in enumerate(sids):
                bits, sizes, _, recon = want[k]
                r = e.result(sid)
                planes = np.concatenate(e.recon(sid))
                assert np.array_equal(planes, recon[i % N]), f"session {k} picture {i}: reconstruction"
                d = clips[k][i % N].astype(np.int64) - planes
                assert r.ssd == tuple(int((p * p).sum()) for p in synth.split(d, W, H)), f"session {k} picture {i}"
                assert (r.levels is not None) == bool(levels)
                if k < sessions:
                    assert r.bits == bits[off[k]:off[k] + sizes[i % N]], f"session {k} picture {i}: bytes"
                    off[k] += sizes[i % N]
                    head = 32 + 26 * 3 + 57 * r.mbs.size
                    assert 0 < r.mbs["coef_bits"].sum() <= 8 * len(r.bits) <= r.mbs["coef_bits"].sum() + head
                else:
                    assert r.bits is None
                    assert not r.mbs["coef_bits"].any()
                assert (r.mbs["quant"] == QUANT).all()
