"""The encoder's timed cases: pictures in, H.261 bitstreams (or macroblock
records, levels and reconstructions) out, through the public entry points.

A case is one kind of caller:

  batch      an engine with many sessions that encodes a few pictures of each
             per pass, three steps in flight, and takes every picture's bytes
             (the batched transcoder; pictures from device or host memory)
  live       an engine whose caller waits for every picture: one step per
             pass, its bytes or its records and levels read before the next
  app        the file encoder's loop for one picture: submit, step, wait,
             bytes, PSNR and reconstruction
  noalloc    h261b_encode_picture_noalloc on the caller's own device buffers
  boundary   the reference's sixteen device calls for one picture, as its
             host code makes them (uploads, motion estimation, host mode
             decision, encode, decode)

Sizes are those of the repository's workloads and plain configurations (QCIF
and CIF, 64 mixed streams, 1024 motion-heavy streams, QUANT 4..24, CBR), and
generic picture sizes for the entry points that write no bitstream.  Sources
are the repository's seeded clips, played forwards and backwards.
"""
import ctypes
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from h261enc_cuda_b200 import _lib, compat, synth, workloads
from h261enc_cuda_b200.engine import Engine

QCIF, CIF = (176, 144), (352, 288)
# what every case has; a listed or drawn case names what differs
DEFAULTS = {"kind": "batch", "qcif": 0, "cif": 0, "width": 0, "height": 0, "pictures": 1, "source": "device",
            "full_search": False, "fmad": True, "quant": 0, "bitrate": 0, "intra_period": 0, "bitstream": True,
            "psnr": False, "levels": False, "motion": False}
# pictures a stream has encoded before the timed passes begin: the engine's
# trial of its launch plan takes its first 27 mostly-inter steps, and the
# steps after it capture their launch graphs
OPENING = 40


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a transcoding node's steady state: 40 QCIF + 24 CIF streams, pictures already on the device
        _case("batch64_device", qcif=40, cif=24, pictures=12),
        # the same streams from host memory, the end-to-end path
        _case("batch64_host", qcif=40, cif=24, pictures=12, source="host"),
        # the largest: 1024 QCIF streams whose blocks move at random (every vector costs a search)
        _case("stress1024_device", qcif=1024, pictures=6, quant=12, motion=True),
        # offline encodes that ask for the exhaustive search
        _case("full_search_qcif64", qcif=64, pictures=4, full_search=True),
        # joining and refreshing streams: every picture intra
        _case("intra_cif16", cif=16, pictures=4, source="host", intra_period=1),
        # a conference server's tick: the ten or so pictures that are due, read at once
        _case("serve_tick", kind="live", qcif=7, cif=3, source="host"),
        # one QCIF call, one picture at a time (the plain QCIF configuration)
        _case("qcif_live", kind="live", qcif=1, source="host", quant=8),
        # the file encoder on CIF at 384 kbit/s with an intra picture every 132 (the plain CIF configuration)
        _case("cif_cbr_app", kind="app", cif=1, source="host", bitrate=384000, intra_period=132, psnr=True),
        # an analysis caller that wants records and levels of pictures of its own size, no bitstream
        _case("vga_levels", kind="live", width=640, height=480, qcif=4, source="host", bitstream=False, levels=True),
        # the smallest call: one QCIF picture between a caller's own buffers
        _case("noalloc_qcif", kind="noalloc", width=176, height=144, quant=8),
        # the same for a large picture
        _case("noalloc_720p", kind="noalloc", width=1280, height=720, quant=12),
        # the reference's host program on this core, CIF
        _case("boundary_cif", kind="boundary", width=352, height=288, quant=10),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _size(rng, most):
    """A picture size in macroblocks, 1 .. `most` of them, any aspect up to 4."""
    n = _log_int(rng, 1, most)
    w = max(1, min(n, int(round((n * 4 ** rng.uniform(-1, 1)) ** 0.5))))
    return 16 * w, 16 * max(1, n // w)


def draw(rng):
    kind = rng.choice(["batch"] * 4 + ["live"] * 3 + ["app", "noalloc", "noalloc", "boundary"])
    q = rng.choice([0, rng.randint(1, 31)])
    if kind == "batch":
        full = rng.random() < 0.2
        n = _log_int(rng, 2, 60 if full else 400)
        cif = rng.randint(0, max(0, n // 3))
        return _case(qcif=n - cif, cif=cif, pictures=rng.randint(1, 4 if full else 12) if n < 100 else 2,
                     source=rng.choice(["device", "host"]), full_search=full, quant=q,
                     bitrate=rng.choice([0, 0, 0, 64000 * rng.randint(1, 16)]), motion=rng.random() < 0.3,
                     intra_period=rng.choice([0, 0, 0, 1, rng.randint(2, 132)]), fmad=rng.random() < 0.85)
    if kind == "live":
        if rng.random() < 0.3:
            w, h = _size(rng, 1500)
            return _case(kind="live", width=w, height=h, qcif=_log_int(rng, 1, 8), source="host", quant=q,
                         bitstream=False, levels=True)
        return _case(kind="live", qcif=_log_int(rng, 1, 24), cif=rng.randint(0, 6), source="host", quant=q,
                     bitrate=rng.choice([0, 0, 64000 * rng.randint(1, 16)]))
    if kind == "app":
        one = rng.random() < 0.5
        return _case(kind="app", qcif=int(one), cif=int(not one), source="host", psnr=True, quant=q,
                     bitrate=0 if q else 64000 * rng.randint(1, 16), intra_period=rng.choice([0, 132]))
    if kind == "noalloc":
        w, h = _size(rng, 4096)
        return _case(kind="noalloc", width=w, height=h, quant=q or 10, full_search=rng.random() < 0.2,
                     fmad=rng.random() < 0.85, motion=rng.random() < 0.3)
    w, h = rng.choice([QCIF, CIF, _size(rng, 1500)])
    return _case(kind="boundary", width=w, height=h, quant=q or 10)


# ------------------------------------------------------------- prepare

def _streams(c, rng):
    """(width, height, QUANT, seed) of every stream of a case."""
    if c["kind"] in ("noalloc", "boundary"):
        sizes = [(c["width"], c["height"])]
    elif c["width"]:
        sizes = [(c["width"], c["height"])] * c["qcif"]
    else:
        sizes = [QCIF] * c["qcif"] + [CIF] * c["cif"]
    return [(w, h, c["quant"] or int(rng.integers(4, 25)), int(rng.integers(1, 2 ** 62))) for w, h in sizes]


def _clips(c, streams, length):
    preset = synth.PRESET_BLOCK_MOTION if c["motion"] else synth.PRESET_STREAM

    def clip(s):
        # a picture smaller than the generator's objects is cut from a larger one
        w, h = max(s[0], 64), max(s[1], 64)
        full = synth.clip(preset, w, h, s[3], length)
        if (w, h) == s[:2]:
            return full
        return np.stack([np.concatenate([p.reshape(-1, w // k)[:s[1] // k, :s[0] // k].ravel()
                                         for p, k in zip(synth.split(f, w, h), (1, 2, 2))]) for f in full])

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        return list(ex.map(clip, streams))


class _EngineState:
    """An engine, its open sessions and their clips, past the streams' opening."""

    def __init__(self, c, seed):
        self.case = c
        streams = _streams(c, np.random.default_rng(seed))
        self.n = len(streams)
        self.length = 4 if self.n > 100 else 8
        clips = _clips(c, streams, self.length)
        mbs = sum(w * h // 256 for w, h, _, _ in streams)
        self.engine = Engine(max_sessions=self.n + 8, me_mode=int(c["full_search"]), fmad=int(c["fmad"]),
                             levels_to_host=int(c["levels"]), bits_host_bytes=max(8 << 20, 512 * mbs))
        cbr = int(c["bitrate"] > 0)
        self.sids = np.array([self.engine.open(w, h, q, intra_period=c["intra_period"], bitstream=int(c["bitstream"]),
                                               rate_control=cbr, bitrate=c["bitrate"], psnr=int(c["psnr"]))
                              for w, h, q, _ in streams], np.int32)
        # every plane 256-byte aligned, all pictures of a stream in one buffer
        ny = [w * h for w, h, _, _ in streams]
        up = lambda v: (v + 255) // 256 * 256   # noqa: E731
        self.planes = []
        if c["source"] == "device":
            rows = []
            for clip, y in zip(clips, ny):
                row = np.zeros((self.length, up(y) + 2 * up(y // 4)), np.uint8)
                row[:, :y] = clip[:, :y]
                row[:, up(y):up(y) + y // 4] = clip[:, y:y + y // 4]
                row[:, up(y) + up(y // 4):up(y) + up(y // 4) + y // 4] = clip[:, y + y // 4:]
                rows.append(row)
            flat = torch.from_numpy(np.concatenate([r.ravel() for r in rows])).cuda()
            at = np.concatenate([[0], np.cumsum([r.size for r in rows])])[:-1] + flat.data_ptr()
            stride = np.array([r.shape[1] for r in rows])
            off_cb = np.array([up(y) for y in ny])
            off_cr = off_cb + np.array([up(y // 4) for y in ny])
            self.keep = flat
        else:
            at = np.array([clip.ctypes.data for clip in clips])
            stride = np.array([clip.shape[1] for clip in clips])
            off_cb = np.array(ny)
            off_cr = off_cb + np.array(ny) // 4
            self.keep = clips
        for i in range(self.length):
            base = at + i * stride
            self.planes.append(tuple(np.ascontiguousarray(a, np.uint64)
                                     for a in (base, base + off_cb, base + off_cr)))
        # the caller's output buffer: room for a pass's bytes (far above what these clips need), zero past them
        self.out = np.zeros(mbs * c["pictures"] * (96 + 600 // (c["quant"] or 4)) if c["bitstream"] else 0, np.uint8)
        self.out_used = 0
        self.queued = 0
        for _ in range(OPENING):
            self.submit()
            self.engine.step()
            self.engine.sync()

    def submit(self):
        """The next picture of every stream."""
        y, cb, cr = self.planes[workloads.clip_index(self.queued, self.length)]
        self.queued += 1
        if self.case["source"] == "device":
            self.engine.submit_device_batch(self.sids, y, cb, cr)
        else:
            self.engine.submit_batch(self.sids, y, cb, cr, wait=False)

    def take(self, at):
        """The latest completed step's pictures, in session order, into the output buffer from byte `at` on; returns
        their sizes and where the next step's go."""
        pics, span = self.engine.step_pictures(self.n + 8)
        if (pics["status"] != 0).any():
            raise RuntimeError("a picture is not in the host arena")
        sizes = pics["bytes"].copy()
        start = pics["bits"].astype(np.int64) - (span.ctypes.data if span.size else 0)
        end = at + int(sizes.sum())
        np.concatenate([span[a:a + b] for a, b in zip(start.tolist(), sizes.tolist())], out=self.out[at:end])
        return sizes, end

    def taken(self, end):
        """The output buffer, which a pass has filled up to `end`."""
        self.out[end:self.out_used] = 0
        self.out_used = end
        return self.out


class _NoallocPicture(ctypes.Structure):   # h261b_noalloc_picture_t, include/h261b.h
    _fields_ = [(n, ctypes.c_int32) for n in ("width", "height", "frame_type", "quant", "me_mode", "fmad", "denoise",
                                              "reset_state")] + \
               [(n, ctypes.c_void_p) for n in ("cur_y", "cur_cb", "cur_cr", "ref_y", "ref_cb", "ref_cr", "rec_y",
                                               "rec_cb", "rec_cr", "state", "mbs", "levels")]


class _NoallocState:
    """A caller's own device buffers: a clip, two reconstructions, the stream's state and results."""

    def __init__(self, c, seed):
        (w, h, q, s), = _streams(c, np.random.default_rng(seed))
        clip, = _clips(c, [(w, h, q, s)], 4)
        self.ny, n = w * h, w * h // 256
        up = lambda v: (v + 255) // 256 * 256   # noqa: E731
        self.off = (0, up(self.ny), up(self.ny) + up(self.ny // 4))
        row = np.zeros((4, self.off[2] + up(self.ny // 4)), np.uint8)
        for i in range(4):
            for o, part in zip(self.off, synth.split(clip[i], w, h)):
                row[i, o:o + part.size] = part
        self.cur = torch.from_numpy(row).cuda()
        self.rec = torch.zeros((2, row.shape[1]), dtype=torch.uint8, device="cuda")
        self.state = torch.zeros(1040, dtype=torch.uint8, device="cuda")   # H261B_NOALLOC_STATE_BYTES
        self.mbs = torch.zeros((n, 16), dtype=torch.uint8, device="cuda")
        self.levels = torch.zeros((n, 384), dtype=torch.int8, device="cuda")
        lib = _lib.core()
        self.call = lib.h261b_encode_picture_noalloc
        self.call.argtypes = [ctypes.POINTER(_NoallocPicture), ctypes.c_void_p]
        self.call.restype = ctypes.c_int32
        self.pic = _NoallocPicture(w, h, 0, q, int(c["full_search"]), int(c["fmad"]), 5, 1)
        self.pic.state, self.pic.mbs, self.pic.levels = (t.data_ptr() for t in (self.state, self.mbs, self.levels))
        self.coded = 0
        self.encode()              # the stream's first picture, intra
        self.pic.frame_type, self.pic.reset_state = _lib.FRAME_TYPE_INTER, 0

    def encode(self):
        k = self.coded
        self.coded += 1
        p = self.pic
        cur = self.cur[workloads.clip_index(k, 4)].data_ptr()
        ref, rec = self.rec[(k + 1) & 1].data_ptr(), self.rec[k & 1].data_ptr()
        p.cur_y, p.cur_cb, p.cur_cr = (cur + o for o in self.off)
        p.ref_y, p.ref_cb, p.ref_cr = (ref + o for o in self.off)
        p.rec_y, p.rec_cb, p.rec_cr = (rec + o for o in self.off)
        _lib.check(self.call(ctypes.byref(p), torch.cuda.current_stream().cuda_stream), "h261b_encode_picture_noalloc")
        return {"recon": self.rec[k & 1], "mbs": self.mbs, "levels": self.levels, "state": self.state}


class _BoundaryState:
    """The process-global encoder behind the reference's calls, and one stream's clip.  Denoise strength 0 leaves no
    state in the encoder from picture to picture, so that several streams of one size can use it in turn."""
    encoder = None

    def __init__(self, c, seed):
        self.case = c
        w, h = c["width"], c["height"]
        streams = _streams(c, np.random.default_rng(seed))
        clip, = _clips(c, streams, 4)
        self.pictures = [tuple(np.ascontiguousarray(p) for p in synth.split(f, w, h)) for f in clip]
        held = _BoundaryState.encoder
        if held is None or (held.w, held.h) != (w, h):
            if held is not None:
                held.close()
            _BoundaryState.encoder = compat.Boundary(w, h, denoise=0)
        self.enc = _BoundaryState.encoder
        self.ref = tuple(np.zeros_like(p) for p in self.pictures[0])
        self.coded = 0
        self.encode()

    def encode(self):
        """One picture in the order of the reference's frame loop (src/h261_main.c:319-365)."""
        first = self.coded == 0
        e = self.enc
        e.set_current(*self.pictures[workloads.clip_index(self.coded, 4)])
        e.set_reference(*self.ref)
        self.coded += 1
        me = e.motion_estimation()
        # the host's mode decision (src/h261_moded.c:53-95)
        md = np.zeros(e.nmb, _lib.MD_DTYPE)
        intra = (me["intra"] <= me["cost"]) & (me["intra"] <= me["fcost"]) | first
        filt = (me["fcost"] < me["cost"]) & ~intra
        moved = ((me["mvx"] != 0) | (me["mvy"] != 0) | filt) & ~intra
        md["type"] = np.where(intra, _lib.MB_TYPE_INTRA, _lib.MB_TYPE_INTER)
        md["flags"] = moved * _lib.MB_MC + filt * _lib.MB_FILTER
        md["mvx"], md["mvy"] = np.where(intra, 0, me["mvx"]), np.where(intra, 0, me["mvy"])
        md["cost"] = np.where(intra, me["intra"], np.where(filt, me["fcost"], me["cost"]))
        mbs = e.encode(md, self.case["quant"], _lib.FRAME_TYPE_INTRA if first else _lib.FRAME_TYPE_INTER)
        self.ref = e.decode()
        return {"me": _bytes_of(me), "mbs": _bytes_of(mbs), "recon": self.ref}


def _bytes_of(a):
    """A structured array as rows of bytes."""
    return np.ascontiguousarray(a).view(np.uint8).reshape(a.size, -1)


class _Result(np.ndarray):
    """An engine's result in its pinned arena, for as long as it is held (the engine is held with it)."""
    engine = None


def _held(a, engine):
    a = a.view(_Result)
    a.engine = engine
    return a


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    kind = {"noalloc": _NoallocState, "boundary": _BoundaryState}.get(c["kind"], _EngineState)
    return kind(c, seed)


# ----------------------------------------------------------------- run

def _batch(st):
    """`pictures` steps, the host reading step k-2 while k-1 and k run."""
    e, first, steps = st.engine, st.queued, st.case["pictures"]
    sizes, end = [], 0
    for k in range(steps + 2):
        if k < steps:
            st.submit()
        if k >= 2:
            e.wait_step(first + k - 2)
            taken, end = st.take(end)
            sizes.append(taken)
        if k < steps:
            e.step()
    _, records = e.step_records()
    return {"sizes": np.concatenate(sizes), "bits": st.taken(end), "records": _held(_bytes_of(records), e)}


def _live(st):
    e = st.engine
    st.submit()
    e.step()
    e.sync()
    _, records = e.step_records()
    out = {"records": _held(_bytes_of(records), e)}
    if st.case["bitstream"]:
        out["sizes"], end = st.take(0)
        out["bits"] = st.taken(end)
    if st.case["levels"]:
        out["levels"] = [_held(e.result(int(s), copy=False).levels, e) for s in st.sids]
    return out


def _app(st):
    """One picture of the file encoder's loop."""
    e, sid = st.engine, int(st.sids[0])
    e.submit_frame(sid, st.keep[0][workloads.clip_index(st.queued, st.length)])
    st.queued += 1
    e.step()
    e.sync()
    r = e.result(sid)
    st.out[:len(r.bits)] = np.frombuffer(r.bits, np.uint8)
    return {"bits": st.taken(len(r.bits)), "size": len(r.bits), "quant": r.quant, "cost": int(r.mbs["cost"].sum()),
            "ssd": list(r.ssd), "recon": e.recon(sid)}


def run(state):
    if isinstance(state, (_NoallocState, _BoundaryState)):
        return state.encode()
    return {"batch": _batch, "live": _live, "app": _app}[state.case["kind"]](state)


# ---------------------------------------------------------------- work

def work(case):
    """Per macroblock: 384 bytes each of source, reference (inter pictures), reconstruction and levels, a 16-byte
    record; one absolute difference and one addition per pixel and vector searched (170 vectors in the reference's
    search, 961 in the exhaustive one, none in intra pictures), and the six blocks' transforms."""
    c = dict(DEFAULTS, **case)
    streams = _streams(c, np.random.default_rng(0))
    mbs = sum(w * h // 256 for w, h, _, _ in streams) * c["pictures"]
    inter = c["intra_period"] != 1
    vectors = (961 if c["full_search"] else 170) if inter else 0
    return {"bytes": mbs * (384 * (4 if inter else 3) + 16), "flops": mbs * (vectors * 512 + 6 * 2 * 16 * 42)}
