"""Learned MV proposer on the GPU (govid_gb300/csrc/mvnet_kernels.cu): the
exhaustive search kernel against brute force, the forward and backward
kernels against the CPU reference (oracle/mvnet_ref.py), one training step,
and the trained net's gain over the same search without it; encodes made
with it decode bit-exact on the GPU and on the oracle."""
import numpy as np
import pytest

import ebiv_oracle
import mvnet_ref as R
from govid_gb300 import ebiv, mvnet

pytestmark = pytest.mark.gpu


def _frames(w, h, seed, n=2):
    sc = ebiv.Scene(mvnet.clip_spec(seed, w, h, sprites=6))
    return [mvnet.luma(sc.render(i), w, h).copy() for i in range(n)]


def _brute(cur, ref, rng):
    H, W = cur.shape
    out = []
    for mby in range(H // 16):
        for mbx in range(W // 16):
            blk = cur[mby * 16: mby * 16 + 16, mbx * 16: mbx * 16 + 16].astype(np.int64)
            best = None
            order = [(0, 0)] + [(dx, dy) for dy in range(-rng, rng + 1) for dx in range(-rng, rng + 1)]
            for dx, dy in order:
                ys = np.clip(np.arange(mby * 16 + dy, mby * 16 + dy + 16), 0, H - 1)
                xs = np.clip(np.arange(mbx * 16 + dx, mbx * 16 + dx + 16), 0, W - 1)
                s = int(np.abs(blk - ref[np.ix_(ys, xs)].astype(np.int64)).sum())
                if best is None or s < best[0]:
                    best = (s, dx, dy)
            out.append(best)
    return out


def test_exhaustive_search_matches_brute_force(gpu_required):
    cur, ref = _frames(64, 48, 21)
    net = mvnet.MvNet(64, 48)
    for rng in (3, 6):
        mv, sad = net.exhaustive(cur, ref, rng)
        want = _brute(cur, ref, rng)
        assert [(int(s), int(x), int(y)) for s, (x, y) in zip(sad, mv)] == want


def _setup(batch=2, seed=5):
    w, h = 64, 48
    net = mvnet.MvNet(w, h, max_batch=batch, seed=seed)
    x0, labs = [], []
    for b in range(batch):
        cur, ref = _frames(w, h, 40 + b)
        lab, _ = net.exhaustive(cur, ref)
        net.set_input(b, cur, ref, lab)
        x0.append(np.stack([R.downsample(cur), R.downsample(ref)]))
        labs.append(lab)
    return net, np.array(x0), np.array(labs)


def test_forward_matches_cpu_reference(gpu_required):
    net, x0, _ = _setup()
    head = net.head(2).astype(np.float64)
    want, _ = R.forward(net.params.astype(np.float64), x0)
    err = np.abs(head - want).max() / np.abs(want).max()
    assert err < 1e-2, err  # BF16 activations; FP32 accumulation order


def test_gradients_match_cpu_reference(gpu_required):
    net, x0, labs = _setup()
    g, stats = net.gradients(2)
    loss, want = R.loss_and_grads(net.params.astype(np.float64), x0, labs)
    assert abs(stats[0] - loss) <= 1e-3 * max(1.0, abs(loss))
    off = 0
    for co, ci in R.SHAPES:
        for n in (co * ci * 9, co):
            a, b = g[off: off + n].astype(np.float64), want[off: off + n]
            rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12)
            assert rel < 2e-2, (off, n, rel)  # tolerance: BF16 activations and weights
            off += n


def test_training_steps_reduce_the_loss(gpu_required):
    net, _, _ = _setup(seed=9)
    first = net.train_step(2, 3e-3)[0]
    for _ in range(30):
        last = net.train_step(2, 3e-3)[0]
    assert last < 0.8 * first


def _hit_rate(net, clips, w=320, h=192):
    """Fraction of macroblocks whose exhaustive-search vector lies within the
    one-pixel neighbourhood of one of the net's 8 proposals."""
    hits = total = 0
    for seed in clips:
        cur, ref = _frames(w, h, seed)
        lab, _ = net.exhaustive(cur, ref)
        cand = net.propose(cur, ref)
        d = np.abs(cand.astype(np.int32) - lab[:, None, :].astype(np.int32)).max(axis=2)
        hits += int((d <= 1).any(axis=1).sum())
        total += lab.shape[0]
    return hits / total


@pytest.fixture(scope="module")
def trained():
    if not mvnet.WEIGHTS.exists():
        pytest.fail(f"{mvnet.WEIGHTS} is missing: train with python -m govid_gb300.train_mvnet")
    return mvnet.MvNet(320, 192).load()


def test_trained_net_gains_over_untrained(gpu_required, trained):
    clips = [9001, 9002, 9003]
    untrained = mvnet.MvNet(320, 192, seed=1)
    got, base = _hit_rate(trained, clips), _hit_rate(untrained, clips)
    assert got > base + 0.2 and got > 0.6, (got, base)


def test_proposed_encode_decodes_bit_exact_and_beats_no_net(gpu_required, trained):
    spec = mvnet.clip_spec(9100, 320, 192, sprites=8)
    sc = ebiv.Scene(spec)
    frames = [sc.render(i) for i in range(6)]
    sizes = {}
    for name in ("proposed", "zero"):
        enc = ebiv.Encoder(ebiv.Config(320, 192), intra=22, gop=6, tiles=(2, 2), search="proposed")
        net = trained if name == "proposed" else mvnet.MvNet(320, 192, seed=1)
        if name == "zero":
            net.params = np.zeros(mvnet.PARAMS, np.float32)  # every proposal falls in the centre bins
        net.attach(enc)
        for f in frames:
            enc.write_frame(f)
        enc.close()
        data = enc.output()
        sizes[name] = len(data)
        pk = [p.data for p in ebiv.Reader(data).packets()]
        want = ebiv_oracle.decode_all(pk)
        c = ebiv.Codec()
        for i, p in enumerate(pk):
            assert c.decode(p).packed() == want[i][1], f"{name} frame {i}"
    assert sizes["proposed"] < sizes["zero"], sizes


@pytest.mark.parametrize("rng", [0, 1, 2, 4, 5, 15, 16])
def test_exhaustive_search_of_any_range(gpu_required, rng):
    """Ranges whose rows of vectors are not whole groups of the kernel's, the smallest and the largest, on noise
    (every vector differs) and on a flat plane (every vector ties)."""
    r = np.random.default_rng(rng)
    net = mvnet.MvNet(48, 32)
    for cur, ref in ((r.integers(0, 256, (32, 48), np.uint8), r.integers(0, 256, (32, 48), np.uint8)),
                     (np.full((32, 48), 255, np.uint8), np.zeros((32, 48), np.uint8))):
        mv, sad = net.exhaustive(cur, ref, rng)
        assert [(int(s), int(x), int(y)) for s, (x, y) in zip(sad, mv)] == _brute(cur, ref, rng)
