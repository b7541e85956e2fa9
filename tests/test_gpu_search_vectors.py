"""The search finds the oracle's vectors where a macroblock's block moved by a
given vector: the corners and edges of [-15, 15]^2, the coarse grid's rows and
columns and their neighbours, in pictures whose border macroblocks have few
vectors.  Integer arithmetic throughout: equality, no tolerance."""
import numpy as np
import pytest

import oracle as O
from h261enc_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu

STEPS = [-15, -14, -13, -3, -2, -1, 0, 1, 2, 3, 13, 14, 15]


@pytest.mark.parametrize("me_mode", [0, 1])
@pytest.mark.parametrize("w,h", [(48, 48), (176, 144)])
def test_known_vectors(gpu, w, h, me_mode):
    rng = np.random.default_rng(w + me_mode)
    # smooth texture, so that the coarse grid leads to the vector's neighbourhood
    base = rng.normal(0, 1, (h + 64, w + 64))
    for _ in range(3):
        base = (base + np.roll(base, 1, 0) + np.roll(base, 1, 1) + np.roll(base, -1, 0) + np.roll(base, -1, 1)) / 5
    base = np.clip(128 + 60 * base / base.std(), 0, 255).astype(np.uint8)
    chroma = np.full(w * h // 2, 128, np.uint8)
    x = y = 32
    frames, vectors = [], [(0, 0)] + [(a, b) for a in STEPS[::2] for b in STEPS[::3]] + [(15, 15), (-15, -15), (0, 0)]
    for vx, vy in vectors:
        # the window moves by the vector; kept inside the texture
        x = x + vx if 0 <= x + vx <= 64 else x - vx
        y = y + vy if 0 <= y + vy <= 64 else y - vy
        frames.append(np.concatenate([base[y:y + h, x:x + w].ravel(), chroma]))
    frames = np.stack(frames)
    want = O.encode_sequence(frames, w, h, 8, me_mode=me_mode)
    with Engine(me_mode=me_mode) as e:
        sid = e.open(w, h, 8)
        for i in range(len(frames)):
            e.submit_frame(sid, frames[i])
            e.step()
            e.sync()
            got = e.result(sid).to_abi(w)
            assert np.array_equal(got["mv"], want["mbs"][i]["mv"]), f"picture {i}: vectors"
            assert np.array_equal(got["tcoeff"], want["mbs"][i]["tcoeff"]), f"picture {i}: levels"
