"""The entropy kernel's symbol chain with its log where the kernel has it, in the macroblocks' coefficient
regions (tests/native/chain_rooms_test.cpp), against the plain decoder, and what a frame's scratch takes."""
import os
import struct
import subprocess

import numpy as np
import pytest

from govid_gb300 import ebiv

from helpers import encode_gen
from test_host_fuzz_cpu import _build, _streams
from test_symbol_chain_cpu import _corrupt


def _packets(data):
    return [p.data for p in ebiv.Reader(data).packets()]


def _full_blocks(qp, mode, seed):
    """A key frame whose macroblocks go from empty to one escape and one sign for every coefficient."""
    rng = np.random.default_rng(seed)
    levels = np.zeros((12, 384), np.int32)
    for m in range(12):
        n = 384 * m // 11
        levels[m, rng.permutation(384)[:n]] = rng.choice([-1, 1], n) * rng.integers(1, 12 if m % 2 else 6, n)
    return ebiv.encode_key_from_levels(64, 48, qp, mode, levels)


def _run(exe, tmp_path, streams):
    blob = struct.pack("<I", len(streams))
    for s in streams:
        blob += struct.pack("<I", len(s)) + b"".join(struct.pack("<I", len(p)) + p for p in s)
    (tmp_path / "streams.bin").write_bytes(blob)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0", UBSAN_OPTIONS="print_stacktrace=1")
    r = subprocess.run([str(exe), str(tmp_path / "streams.bin")], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stdout + r.stderr[-4000:]
    f = r.stdout.split()
    return dict(zip(f[0::2], map(int, f[1::2])))


def test_logs_in_the_coefficient_regions(tmp_path):
    exe = _build(tmp_path, "chain_rooms_test", ("payload.cpp", "container.cpp"))
    rng = np.random.default_rng(7)
    streams = _streams(seed=12, per_clip=8)
    for w, h, q, tiles in [(64, 48, 4, (1, 1)), (37, 21, 20, (2, 1)), (160, 96, 12, (2, 2)), (16, 16, 0, (1, 1)),
                           (96, 64, 20, (6, 4)), (320, 192, 22, (20, 12))]:
        streams.append(_packets(encode_gen(w, h, 5, ebiv.synth_pan, intra=q, gop=5, tiles=tiles)[0]))
    streams += [_corrupt(s, rng) for s in streams for _ in range(6)]
    for q in (0, 4, 8):
        spec = ebiv.SceneSpec(width=320, height=192, seed=5, sprites=6, noise_y16=60, noise_c16=30)
        streams.append(_packets(ebiv.encode_scene(spec, 3, qp=q, gop=3, tiles=(2, 1), fast=True, threads=4)))
    streams += [[_full_blocks(20, m, s)] for m in range(2) for s in range(4)]
    got = _run(exe, tmp_path, streams)
    # Small tiles too (of up to six macroblocks, which a log by the tile has no room for), macroblocks that do not
    # fit and tiles that end at an error, both of which leave everything else to the chain.
    assert got["compared"] > 8000 and got["small"] > 6000 and got["logged"] > 50000, got
    assert got["failing"] > 1000 and got["stopped"] > 300 and got["dense"] > 100 and got["resumed"] > 300, got


@pytest.mark.parametrize("w,h", [(1, 1), (16, 16), (37, 21), (160, 96), (640, 360), (1280, 720), (1920, 1080), (8192, 4320)])
@pytest.mark.parametrize("lookahead", [1, 4, 32, 64])
def test_a_stream_takes_no_more_memory(w, h, lookahead):
    """A stream's frames take their macroblocks' records, coefficient regions and lists and no more than 1909 bytes a
    macroblock, whatever the size (a server admits streams by this figure)."""
    cols, rows = (w + 15) // 16, (h + 15) // 16
    align = lambda v: (v + 63) // 64 * 64  # noqa: E731
    frame = align(16 * cols) * 16 * rows + 2 * align(8 * cols) * 8 * rows
    pool = 3 + 2 * lookahead + 3
    assert ebiv.stream_footprint(w, h, 3, lookahead) <= pool * frame + (lookahead + 1) * 1909 * cols * rows
