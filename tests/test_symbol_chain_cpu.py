"""The entropy kernel's symbol chain, compiled for the host with sanitizers, against a
plain restatement of the decoder (tests/native/chain_test.cpp): intact clips of every
transform size and both frame types, and seeded mutations of the tile bytes."""
import os
import struct
import subprocess

import numpy as np

from govid_gb300 import ebiv

from helpers import encode_gen
from test_host_fuzz_cpu import _build, _streams


def _corrupt(stream, rng):
    """Tile bytes flipped, cut or cleared (the tables and lengths in front of them mostly stay)."""
    out = []
    for p in stream:
        b = bytearray(p)
        at = int(rng.integers(min(len(b), 150), len(b) + 1))
        kind = int(rng.integers(0, 4))
        if kind == 0 and at < len(b):
            b[at] ^= 1 << int(rng.integers(0, 8))
        elif kind == 1:
            b[at:] = bytes(len(b) - at)
        elif kind == 2 and at < len(b):
            b[at] = int(rng.integers(0, 256))
        out.append(bytes(b))
    return out


def test_chain_equals_the_plain_decoder(tmp_path):
    exe = _build(tmp_path, "chain_test", ("payload.cpp", "container.cpp"))
    rng = np.random.default_rng(7)
    streams = _streams(seed=11, per_clip=8)
    for w, h, q, tiles in [(64, 48, 4, (1, 1)), (37, 21, 20, (2, 1)), (160, 96, 12, (2, 2)), (16, 16, 0, (1, 1))]:
        data, _, _ = encode_gen(w, h, 5, ebiv.synth_pan, intra=q, gop=5, tiles=tiles)
        streams.append([p.data for p in ebiv.Reader(data).packets()])
    streams += [_corrupt(s, rng) for s in streams for _ in range(6)]
    # Enough symbols of low frequency for states that take two bytes at every place of the chain's loop.
    spec = ebiv.SceneSpec(width=640, height=368, seed=5, sprites=6, noise_y16=60, noise_c16=30)
    data = ebiv.encode_scene(spec, 3, qp=8, gop=3, tiles=(1, 1), fast=True, threads=4)
    streams.append([p.data for p in ebiv.Reader(data).packets()])
    blob = struct.pack("<I", len(streams))
    for s in streams:
        blob += struct.pack("<I", len(s)) + b"".join(struct.pack("<I", len(p)) + p for p in s)
    (tmp_path / "streams.bin").write_bytes(blob)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0", UBSAN_OPTIONS="print_stacktrace=1")
    r = subprocess.run([str(exe), str(tmp_path / "streams.bin")], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stdout + r.stderr[-4000:]
    f = r.stdout.split()
    counts = dict(zip(f[0::2], map(int, f[1::2])))
    assert counts["tiles"] > 2000 and counts["failing"] > 100 and counts["overflowing"] > 20, counts
