"""What the entropy stage costs where it is not in its ordinary course, against that course on the same tile."""
import ctypes as C
import statistics
import time

import numpy as np
import pytest

import ebiv_oracle
from govid_gb300 import _native, ebiv

from helpers import encode_gen

pytestmark = pytest.mark.gpu

W, H = 640, 368


def _key(seed=3, most=60, full=(), least=3):
    """A key frame of one tile, about 100 symbols a macroblock: its chain is nearly all of its decode's time.  The
    macroblocks of `full` have all of their coefficients and many escapes, more than their log has room for."""
    rng = np.random.default_rng(seed)
    mbs = (W // 16) * (H // 16)
    levels = np.zeros((mbs, 384), np.int32)
    at = rng.integers(0, 384, (mbs, most))
    levels[np.arange(mbs)[:, None], at] = rng.integers(-3, 4, (mbs, most))
    for m in full:
        levels[m] = rng.choice([-1, 1], 384) * rng.integers(least, 9, 384)
    return ebiv.encode_key_from_levels(W, H, 20, 0, levels)


def _status(codec, pkt):
    try:
        codec.decode(pkt)
        return 0
    except ebiv.EbivError as e:
        return e.status


def _ms(f, n=7):
    f()
    took = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        took.append(1000 * (time.perf_counter() - t0))
    return statistics.median(took)


def test_key_frames_without_allocation_take_the_time_of_the_codec(gpu_required):
    # Both are synchronous calls and wait for one chain; the codec copies the frame to the host as well.  Decoded by
    # the full chain a key frame takes 2.5 times the chain's time and more.
    import torch

    pkt = _key()
    y = torch.empty(W * H, dtype=torch.uint8, device="cuda")
    cb, cr = (torch.empty(W * H // 4, dtype=torch.uint8, device="cuda") for _ in range(2))
    w, h = C.c_int32(), C.c_int32()

    def noalloc():
        assert _native.lib().ebivgpu_decode_key_noalloc(pkt, len(pkt), y.data_ptr(), W, W * H, cb.data_ptr(),
                                                        cr.data_ptr(), W // 2, W * H // 4, None, C.byref(w), C.byref(h)) == 0

    codec = ebiv.Codec()
    a, b = _ms(noalloc), _ms(lambda: codec.decode(pkt))
    assert a < 1.5 * b, f"no allocation {a:.2f} ms, codec {b:.2f} ms"
    assert b"".join(p.cpu().numpy().tobytes() for p in (y, cb, cr)) == ebiv_oracle.decode_all([pkt])[0][1]


def _cut(pkt, n):
    """The packet, of one tile, without the tile's first n bytes: read backwards, it fails near its end."""

    def varint(v):
        out = bytearray()
        while v >= 128:
            out.append(v & 127 | 128)
            v >>= 7
        return bytes(out) + bytes([v])

    for at in range(6, 2000):
        size = len(pkt) - at - 3
        if pkt[at:at + 3] == varint(size):
            return pkt[:at] + varint(size - n) + pkt[at + 3 + n:]
    raise AssertionError("no tile")


@pytest.mark.parametrize("what", ["error", "full"])
def test_what_the_chain_leaves_costs_one_pass_more(gpu_required, what):
    # A tile with an error and tiles with macroblocks that have no room for their log: a second pass of the symbol
    # chain and these macroblocks by the full chain, which for a whole tile takes 2.5 passes by itself.
    plain = _key()
    pkt = _cut(plain, 100) if what == "error" else _key(full=(0, 17, 460, 461, 915))
    codec = ebiv.Codec()
    intact, other = _ms(lambda: codec.decode(plain)), _ms(lambda: _status(codec, pkt))
    assert other < 2.5 * intact, f"intact {intact:.2f} ms, {what} {other:.2f} ms"
    st, planes = ebiv_oracle.decode_all([pkt])[0]
    assert _status(codec, pkt) == st == (ebiv.ErrCorrupt.status if what == "error" else 0)
    if st == 0:
        assert codec.decode(pkt).packed() == planes


def test_full_macroblocks_in_a_row_are_not_tried_one_by_one(gpu_required):
    # 920 macroblocks of 384 escapes each: the full chain by itself takes 11.2 times the time of the symbol chain for
    # the plain frame; 14.2 times when every macroblock is tried by the symbol chain first.  In between lies 12.7.
    codec = ebiv.Codec()
    plain, full = _key(), _key(full=range((W // 16) * (H // 16)), least=5)
    a, b = _ms(lambda: codec.decode(plain)), _ms(lambda: codec.decode(full), 3)
    assert b < 12.7 * a, f"plain {a:.2f} ms, full {b:.2f} ms"
    assert codec.decode(full).packed() == ebiv_oracle.decode_all([full])[0][1]


@pytest.mark.parametrize("lookahead,depth", [(1, 0), (4, 0), (4, 2)])
def test_more_jobs_than_ctas_of_several_frames(gpu_required, lookahead, depth):
    # 1000 tiles a frame are 250 entropy jobs; four frames at once have 1000 for the 304 CTAs, which keep a frame's
    # tables from one job to the next and change them with the frame.
    cont, _, _ = encode_gen(640, 400, 8, ebiv.synth_pan, intra=14, gop=3, tiles=(40, 25), keep_recon=False)
    pkts = [p.data for p in ebiv.Reader(cont).packets()]
    want = ebiv_oracle.decode_all(pkts)
    b = ebiv.Batch(lookahead=lookahead, pipeline=depth)
    b.add_stream(pkts)
    got = {}
    for _ in range(len(pkts) + depth + 2):
        for r in b.round():
            got[r.frame_index] = (r.status, b.download(r, 640, 400))
    for r in b.drain():
        got[r.frame_index] = (r.status, b.download(r, 640, 400))
    assert [got[i] for i in range(len(pkts))] == want


def _damaged(stream, rng):
    """Tile bytes of some packets flipped, cleared or replaced (the tables in front of them mostly stay)."""
    out = []
    for p in stream:
        b = bytearray(p)
        at = int(rng.integers(min(len(b) - 1, 150), len(b)))
        kind = int(rng.integers(0, 4))
        if kind == 0:
            b[at] ^= 1 << int(rng.integers(0, 8))
        elif kind == 1:
            b[at:] = bytes(len(b) - at)
        elif kind == 2:
            n = len(b[at:at + 30])
            b[at:at + n] = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
        out.append(bytes(b))
    return out


@pytest.mark.parametrize("q,tiles", [(0, (1, 1)), (2, (2, 2)), (6, (2, 1))])
def test_left_macroblocks_and_errors_match_the_oracle(gpu_required, q, tiles):
    # High quality: macroblocks with and without room for their log beside one another, in key and inter frames;
    # then with damaged tiles, whose errors come before, in and behind such macroblocks.
    rng = np.random.default_rng(40 + q)
    spec = ebiv.SceneSpec(width=160, height=96, seed=5 + q, sprites=6, noise_y16=90, noise_c16=60)
    cont = ebiv.encode_scene(spec, 5, qp=q, gop=4, tiles=tiles, fast=True, threads=4)
    clip = [p.data for p in ebiv.Reader(cont).packets()]
    failing = 0
    for k in range(16):
        pkts = clip if k == 0 else _damaged(clip, rng)
        want = [(st, planes if st == 0 else None) for st, planes in ebiv_oracle.decode_all(pkts)]
        failing += sum(st != 0 for st, _ in want)
        codec = ebiv.Codec()
        assert [_status(codec, p) for p in pkts] == [st for st, _ in want], k
        b = ebiv.Batch(lookahead=3, pipeline=k % 2)
        b.add_stream(pkts)
        res = {}
        for _ in range(3 * len(pkts) + 6):
            for r in b.round():
                res[r.frame_index] = (r.status, b.download(r, 160, 96) if r.status == 0 else None)
        for r in b.drain():
            res[r.frame_index] = (r.status, b.download(r, 160, 96) if r.status == 0 else None)
        assert [res[i] for i in range(len(pkts))] == want, k
    assert failing > 10
