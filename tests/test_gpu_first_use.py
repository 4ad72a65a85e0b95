"""The first decodes of a process, on several threads at once.

Every kernel variant's shared-memory limit is raised on its first use per device; a decode
that starts on another thread meanwhile must not launch before that is done.  Run in fresh
processes, because a process has one first use."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

# One-tile 720p key frames: the intra stage's launch needs the raised limit (16 warps'
# scratch, 7200 progress bytes and the ordering of 3600 macroblocks: over 48 KB).
CODE = """
import sys, threading
sys.path.insert(0, %r)
import numpy as np
from govid_gb300 import ebiv
levels = np.zeros((3600, 384), np.int32)
levels[:, ::16] = np.arange(3600)[:, None] %% 5 - 2
pkt = ebiv.encode_key_from_levels(1280, 720, 20, 0, levels)
codecs = [ebiv.Codec() for _ in range(12)]
gate, got = threading.Barrier(len(codecs)), [None] * len(codecs)
def first(i):
    gate.wait()
    try:
        got[i] = codecs[i].decode(pkt).packed()
    except ebiv.EbivError as e:
        got[i] = e.status
threads = [threading.Thread(target=first, args=(i,)) for i in range(len(codecs))]
[t.start() for t in threads]
[t.join() for t in threads]
bad = [g for g in got if not isinstance(g, bytes) or g != codecs[0].decode(pkt).packed()]
print("bad", [g if isinstance(g, int) else "bytes" for g in bad])
sys.exit(1 if bad else 0)
""" % str(ROOT)


@pytest.mark.parametrize("attempt", range(4))
def test_first_decodes_on_many_threads(gpu_required, attempt):
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
