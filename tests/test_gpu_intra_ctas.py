"""The intra stage with a given number of warps, where a tile has a CTA for luma and one for chroma (up to 76 tiles on
152 SMs) and where one CTA does both."""
import pytest

import ebiv_oracle
from govid_gb300 import ebiv

from helpers import encode_gen, flash_gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [4, 8, 16])
@pytest.mark.parametrize("w,h,grid", [(213, 149, (1, 1)), (213, 149, (3, 2)), (400, 336, (11, 7))])
@pytest.mark.parametrize("qp", [8, 30])
def test_given_warps(gpu_required, warps, w, h, grid, qp):
    # Key frames, and inter frames with intra macroblocks (the picture changes); 77 tiles are one CTA each.
    cont, _, _ = encode_gen(w, h, 4, flash_gen, intra=qp, gop=3, tiles=grid, keep_recon=False)
    pkts = [p.data for p in ebiv.Reader(cont).packets()]
    want = ebiv_oracle.decode_all(pkts)
    assert all(st == 0 for st, _ in want)
    b = ebiv.Batch(lookahead=2, pipeline=1)
    b.set_tuning(2, warps)
    b.add_stream(pkts)
    got = {}
    for _ in range(len(pkts) + 4):
        for r in b.round():
            got[r.frame_index] = (r.status, b.download(r, w, h))
    for r in b.drain():
        got[r.frame_index] = (r.status, b.download(r, w, h))
    assert [got[i] for i in range(len(pkts))] == want
