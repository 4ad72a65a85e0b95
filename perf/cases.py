"""What is timed when the speed of this framework is compared between two of its versions.

Twelve cases of the work that its users have it do, through the public entry points of
``govid_gb300``: the Codec contract (one packet in, one host frame out), the Batch API
(many frames in flight, packets from pinned memory, frames to pinned memory), the
decode-ahead source of a player, scrubbing in a container on the GPU, and the
encoder-side operators (alt-ref filter, block transform, motion search, motion proposer).
Frame sizes, tile grids, quantizers and scene parameters are those of
``govid_gb300/workloads.py``, ``bench.py`` and the tests, or generic video sizes.

Streams are edits of short clips: each geometry has a few groups of pictures, encoded
once per process from fixed scene seeds, and a case's seed draws which of them follow one
another and where each is cut.  The encoder takes 0.1 s of 16 cores and more per 1080p
frame, so that fresh clips for every seed would take longer than everything else.

Every output is whole bytes or whole numbers (decoded planes, RGBA, indexes, transform
coefficients, motion vectors), the same for every correct implementation.
"""
from __future__ import annotations

import math
import os
import random
import struct
import threading
import zlib

import numpy as np
import torch

from govid_gb300 import ebiv
from govid_gb300 import mvnet as _mvnet


def listed():
    return [
        # The smallest calls: a thumbnail-sized one-tile clip through the Codec contract,
        # eight synchronous calls, where the latency of one call is everything.
        dict(name="codec_160x96", kind="codec", w=160, h=96, cols=1, rows=1, qp=22, frames=8, rgba=False, altref=0),
        # A player that decodes one frame per call, ordinary size and grid, with the
        # encoder's alt-ref option (golden override payloads in the key frames).
        dict(name="codec_720p", kind="codec", w=1280, h=720, cols=2, rows=2, qp=22, frames=12, rgba=False, altref=4),
        # The same at 1080p with RGBA output (govid's WithRGBA), the flagship tile grid.
        dict(name="codec_1080p_rgba", kind="codec", w=1920, h=1080, cols=4, rows=3, qp=22, frames=12, rgba=True,
             altref=0),
        # The flagship: one 1080p stream end to end through pipelined rounds.
        dict(name="batch_1080p", kind="batch", sizes="1920x1080:4x3:22", streams=1, frames=96, lookahead=32, depth=3),
        # Many streams of mixed sizes and grids at once (a transcoding or wall server).
        dict(name="batch_mix", kind="batch", sizes="640x360:1x1:28,1280x720:2x2:22,1920x1080:4x3:22", streams=24,
             frames=16, lookahead=4, depth=2),
        # One-tile streams, high quality, one synchronous round per frame time: latency bound.
        dict(name="batch_live_1tile", kind="batch", sizes="1280x720:1x1:18", streams=8, frames=8, lookahead=1, depth=0),
        # An odd-sized small stream, whole clip in a few synchronous rounds.
        dict(name="batch_odd", kind="batch", sizes="853x479:2x2:20", streams=2, frames=20, lookahead=8, depth=0),
        # govid's AsyncPlayer: a consumer that takes a 1080p clip with RGBA from the source.
        dict(name="source_1080p_rgba", kind="source", w=1920, h=1080, cols=4, rows=3, qp=22, frames=16, ahead=8),
        # Scrubbing: seeks resolved on the GPU, one key frame decoded in place after each.
        dict(name="scrub_720p", kind="scrub", w=1280, h=720, cols=2, rows=2, qp=22, seeks=12),
        # The encoder's alt-ref filter over a window of 1080p frames.
        dict(name="altref_1080p", kind="altref", w=1920, h=1080, window=8),
        # forwardDCT and satd of the 8x8 luma blocks of one 1080p frame.
        dict(name="fdct_1080p", kind="fdct", n=8, count=32400),
        # Motion for the encoder's search="proposed": the net's candidates for a 1080p pair,
        # and the exhaustive search that labels its training pairs.
        dict(name="motion_1080p", kind="motion", w=1920, h=1088, range=16),
    ]


_SIZES = [(37, 21), (64, 48), (160, 96), (161, 91), (320, 192), (426, 240), (640, 360), (853, 479), (854, 480),
          (960, 540), (1023, 577), (1280, 720), (1281, 719), (1600, 900), (1920, 1080)]
_GRIDS = [(1, 1), (2, 1), (2, 2), (4, 3)]
_QPS = [18, 20, 22, 28, 32]


def draw(rng):
    kind = rng.choice(["codec", "codec", "batch", "batch", "source", "scrub", "altref", "fdct", "motion"])
    w, h = rng.choice(_SIZES)
    w, h = max(1, w - rng.randrange(0, 9)), max(1, h - rng.randrange(0, 9))
    cols, rows = rng.choice(_GRIDS)
    qp = rng.choice(_QPS)
    if kind == "codec":
        return dict(kind=kind, w=w, h=h, cols=cols, rows=rows, qp=qp, frames=rng.randint(1, 12),
                    rgba=rng.random() < 0.5, altref=rng.choice([0, 0, 4]))
    if kind == "batch":
        return dict(kind=kind, sizes="%dx%d:%dx%d:%d" % (w, h, cols, rows, qp), streams=rng.randint(1, 8),
                    frames=rng.randint(3, 24), lookahead=rng.choice([1, 2, 4, 8, 16]), depth=rng.randint(0, 3))
    if kind == "source":
        return dict(kind=kind, w=w, h=h, cols=cols, rows=rows, qp=qp, frames=rng.randint(2, 16), ahead=8)
    if kind == "scrub":
        return dict(kind=kind, w=w, h=h, cols=cols, rows=rows, qp=qp, seeks=rng.randint(1, 16))
    if kind == "altref":
        return dict(kind=kind, w=w, h=h, window=rng.randint(2, 9))
    if kind == "fdct":
        return dict(kind=kind, n=rng.choice([4, 8, 16]), count=int(math.exp(rng.uniform(math.log(33), math.log(32768)))))
    return dict(kind=kind, w=16 * rng.randint(4, 120), h=16 * rng.randint(4, 67), range=rng.choice([4, 7, 16]))


# ---------------------------------------------------------------------------
# Content
# ---------------------------------------------------------------------------

_GOPS: dict[tuple, list[list[bytes]]] = {}
_LOCK = threading.Lock()


def _gops(w, h, cols, rows, qp, altref=0):
    """Groups of pictures of one geometry: a key frame and its inter frames each.

    Long enough that most frames are inter frames, as in real streams, within a bound on
    the encoder's time (it runs tiles and groups of pictures in parallel)."""
    key = (w, h, cols, rows, qp, altref)
    with _LOCK:
        if key not in _GOPS:
            mbs = ((w + 15) // 16) * ((h + 15) // 16)
            tile = max(1, mbs // min(mbs, cols * rows))
            gop = max(2, min(16, 12000 // tile))
            groups = 2 if gop >= 8 else 4
            spec = ebiv.SceneSpec(width=w, height=h, seed=2024 + w, sprites=6 if w <= 640 else (12 if w <= 1280 else 24),
                                  vel_max_q=16, integer_vel=True, noise_y16=32, noise_c16=16)
            data = ebiv.encode_scene(spec, gop * groups, qp=qp, gop=gop, tiles=(cols, rows), fast=True,
                                     threads=max(1, os.cpu_count() or 1), altref=altref)
            got = []
            for p in ebiv.Reader(data).packets():
                if p.keyframe:
                    got.append([])
                got[-1].append(p.data)
            _GOPS[key] = got
        return _GOPS[key]


def _stream(rng, frames, geometry):
    """`frames` packets: groups of pictures of the geometry in a drawn order, each cut at a drawn length."""
    gops, out = _gops(*geometry), []
    while len(out) < frames:
        g = rng.choice(gops)
        out += g[: rng.randint((len(g) + 1) // 2, len(g))]
    return out[:frames]


def _container(packets, w, h, cols, rows):
    """An EBIV file of these packets (header, frame records, index, footer)."""
    head = b"EBIV" + struct.pack("<HHIIIII4BHHI", 4, 48, w, h, 30, 1, len(packets), 0, 0, 0, 0, cols, rows, 0)
    body, index, at = [head.ljust(48, b"\0")], [], 48
    for p in packets:
        key = 1 if p[0] & 3 == 0 else 0
        body.append(struct.pack("<HHI", 0xEB17, key, len(p)) + p)
        index.append(struct.pack("<QII", at, len(p), key))
        at += 8 + len(p)
    index = b"".join(index)
    return b"".join(body) + index + struct.pack("<QII4s", at, len(packets), zlib.crc32(index), b"EBIX")


def _parse(sizes):
    out = []
    for s in sizes.split(","):
        size, grid, qp = s.split(":")
        out.append((*map(int, size.split("x")), *map(int, grid.split("x")), int(qp)))
    return out


def _frames(seed, w, h, n, hold):
    """Rendered frames, packed; with `hold` a still scene under noise, as in front of an alt-ref."""
    scene = ebiv.Scene(ebiv.SceneSpec(width=w, height=h, seed=1 + seed % (1 << 20), sprites=24, vel_max_q=8 if hold else 32,
                                      integer_vel=False, pan_max_q=0 if hold else 12, noise_y16=16, noise_c16=8))
    return [scene.render(i) for i in range(n)]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind in ("codec", "source", "scrub"):
        geo = (case["w"], case["h"], case["cols"], case["rows"], case["qp"])
    if kind == "codec":
        pkts = [ebiv.Packet(p) for p in _stream(rng, case["frames"], geo + (case["altref"],))]
        codec = ebiv.Codec(ring=case["frames"])  # every frame of a pass stays valid until the next
        codec.with_rgba(case["rgba"])
        return dict(case, pkts=pkts, codec=codec)
    if kind == "batch":
        geos = _parse(case["sizes"])
        b = ebiv.Batch(lookahead=case["lookahead"], pipeline=case["depth"])
        streams, at = {}, 0
        for i in range(case["streams"]):
            g = geos[i % len(geos)]
            pkts = _stream(rng, case["frames"], g)
            pin = torch.frombuffer(bytearray(b"".join(pkts)), dtype=torch.uint8).pin_memory()
            addrs, o = [], pin.data_ptr()
            for p in pkts:
                addrs.append(o)
                o += len(p)
            fb = ebiv.packed_size(g[0], g[1])
            streams[b.add_stream(pkts)] = (pin, addrs, [len(p) for p in pkts], at, fb)
            at += fb * len(pkts)
        return dict(case, b=b, by_id=streams, out=torch.empty(at, dtype=torch.uint8, pin_memory=True))
    if kind == "source":
        pkts = _stream(rng, case["frames"], geo)
        return dict(case, held=[], src=ebiv.AsyncSource(_container(pkts, *geo[:4]), depth=case["ahead"], rgba=True))
    if kind == "scrub":
        pkts = _stream(rng, 64, geo)
        c = ebiv.DeviceContainer(_container(pkts, *geo[:4]))
        b = ebiv.Batch()
        fb = ebiv.packed_size(case["w"], case["h"])
        return dict(case, c=c, b=b, sid=b.add_container(c), fb=fb, times=[rng.randrange(64 * 10**9 // 30) for _ in range(case["seeks"])],
                    out=torch.empty((case["seeks"], fb), dtype=torch.uint8, pin_memory=True))
    if kind == "altref":
        return dict(case, frames=_frames(seed, case["w"], case["h"], case["window"], True), op=ebiv.AltRef())
    if kind == "fdct":
        r = np.random.default_rng(seed)
        blocks = np.clip(np.rint(r.laplace(0, 12, (case["count"], case["n"], case["n"]))), -255, 255).astype(np.int32)
        return dict(case, blocks=blocks, op=ebiv.BlockAnalysis())
    ref, cur = (_mvnet.luma(f, case["w"], case["h"]) for f in _frames(seed, case["w"], case["h"], 2, False))
    return dict(case, cur=cur, ref=ref, net=_mvnet.MvNet(case["w"], case["h"]).load())


class _Views(list):
    """Frames as views of their decoder's memory, and that decoder (`owner`), so that they outlive the state."""

    def __init__(self, frames, owner):
        super().__init__(frames)
        self.owner = owner


def run(s):
    kind = s["kind"]
    if kind == "codec":
        c = s["codec"]
        frames = [c.decode(p) for p in s["pkts"]]
        out = _Views(((f.y, f.cb, f.cr) for f in frames), c)
        # The pooled RGBA of the newest frame, the one on screen.
        return (out, c.pooled_rgba(frames[-1])) if s["rgba"] else out
    if kind == "batch":
        b, by_id, base = s["b"], s["by_id"], s["out"].data_ptr()
        left = 0
        for sid, (_, addrs, lens, _, _) in by_id.items():
            b.reload(sid, addrs, lens)
            left += len(lens)
        while left:
            for r in b.round():
                _, _, _, at, fb = by_id[r.stream]
                if r.status:
                    raise RuntimeError("frame %d of stream %d: status %d" % (r.frame_index, r.stream, r.status))
                b.download_async(r, base + at + r.frame_index * fb, fb)
                left -= 1
        b.drain()
        b.sync()
        return s["out"]
    if kind == "source":
        src = s["src"]
        for f in s["held"]:
            src.release(f)
        src.seek(0)
        s["held"] = [src.next() for _ in range(s["frames"])]
        return _Views(((f.y, f.cb, f.cr, f.rgba) for f in s["held"]), src)
    if kind == "scrub":
        c, b, sid, out, landed = s["c"], s["b"], s["sid"], s["out"], []
        for i, t in enumerate(s["times"]):
            frame, when = c.seek(t)
            b.seek(sid, frame)
            (r,) = b.round()
            if r.status:
                raise RuntimeError("frame %d: status %d" % (frame, r.status))
            b.download_async(r, out[i].data_ptr(), s["fb"])
            landed += [frame, when]
        b.sync()
        return out, np.array(landed, np.int64)
    if kind == "altref":
        got = s["op"].build(s["frames"], s["w"], s["h"], s["window"])
        return np.zeros(0, np.uint8) if got is None else np.frombuffer(got, np.uint8)
    if kind == "fdct":
        return s["op"].fdct_satd(s["blocks"])
    return s["net"].propose(s["cur"], s["ref"]), s["net"].exhaustive(s["cur"], s["ref"], s["range"])


def work(case):
    """Packets once (about 0.002 bytes a sample), one reference sample read and one output sample
    written for each decoded one, and the copy to the host; what the operators read and write."""
    kind = case["kind"]
    if kind in ("codec", "source"):
        n = ebiv.packed_size(case["w"], case["h"])
        rgba = 4 * case["w"] * case["h"] if kind == "source" or case.get("rgba") else 0
        return {"bytes": case["frames"] * (3.002 * n + 2 * rgba), "flops": 0}
    if kind == "batch":
        geos = _parse(case["sizes"])
        n = sum(ebiv.packed_size(*geos[i % len(geos)][:2]) for i in range(case["streams"]))
        return {"bytes": 3.002 * n * case["frames"], "flops": 0}
    if kind == "scrub":
        return {"bytes": case["seeks"] * 2.01 * ebiv.packed_size(case["w"], case["h"]), "flops": 0}
    if kind == "altref":
        return {"bytes": (case["window"] + 1) * ebiv.packed_size(case["w"], case["h"]), "flops": 0}
    if kind == "fdct":
        n = case["n"]
        return {"bytes": case["count"] * (8 * n * n + 8), "flops": case["count"] * 4 * n**3}
    px, mbs = case["w"] * case["h"], (case["w"] // 16) * (case["h"] // 16)
    conv = 2 * 9 * (2 * 32 + 2 * 32 * 32 + 32 * 34) * (px // 16)
    return {"bytes": 4 * px + mbs * 40, "flops": conv + mbs * (2 * case["range"] + 1) ** 2 * 256 * 2}


def exact(case, seed):
    """Every output is whole bytes or whole numbers: there is nothing to measure an error of."""
    return None
