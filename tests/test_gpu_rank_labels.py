"""Rank labels of large groups: groups of more than 2048 suffixes that lose members in some rounds, stand in others and
split near their label's end, against the oracle (U, sampled indexes, suffix array). Periodic texts with flipped bytes
shed a few members a round; runs and repeats of random stretches split groups anywhere; batches give groups of several
blocks to one bucket pass. With the radix round 0 (raw and coded keys) and with the bucket passes' own round 0."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


def _text(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind.startswith("period"):
        p = int(kind[6:])
        t = np.resize(rng.integers(97, 123, p).astype(np.uint8), n)
        for q in rng.integers(0, n, max(2, n // 20000)):
            t[q] ^= int(rng.integers(1, 256))
        return t
    if kind == "runs":  # long runs of two values
        return np.repeat(rng.integers(0, 2, n).astype(np.uint8), rng.integers(1, 400, n))[:n].copy()
    if kind == "copies":  # one stretch over and over, cut at random lengths
        s = rng.integers(0, 4, 3000).astype(np.uint8)
        out = []
        while sum(map(len, out)) < n:
            out.append(s[int(rng.integers(0, 500)):int(rng.integers(600, 3000))])
        return np.concatenate(out)[:n].copy()
    a, b = np.array([97], np.uint8), np.array([97, 98], np.uint8)
    while b.size < n:
        a, b = b, np.concatenate([b, a])
    return b[:n].copy()


@pytest.mark.parametrize("kind", ["period1", "period3", "period64", "period4097", "runs", "copies", "fibonacci"])
@pytest.mark.parametrize("lsd_round0,lsd_bytes", [(1, 8), (1, 16), (0, 16)])
def test_large_groups_keep_or_change_their_label(kind, lsd_round0, lsd_bytes):
    import torch

    sizes = [2049, 40_000, 300_001, 4096]
    texts = [_text(kind, n, n + k) for k, n in enumerate(sizes)]
    offs, off = [], 0
    for t in texts:
        offs.append(off)
        off += (t.size + 15) // 16 * 16
    buf = np.zeros(off + 64, np.uint8)
    for t, o in zip(texts, offs):
        buf[o:o + t.size] = t
    r, iouts, k = 1 << 8, [], 0
    for t in texts:
        iouts.append(k)
        k += (t.size - 1) // r + 1
    dT = torch.from_numpy(buf).cuda()
    dL = torch.zeros(off + len(texts), dtype=torch.uint8, device="cuda")
    dI = torch.zeros(k, dtype=torch.int32, device="cuda")
    dSA = torch.zeros(off, dtype=torch.int32, device="cuda")
    eng = codec.Engine()
    eng.config(lsd_round0=lsd_round0, lsd_bytes=lsd_bytes)
    blocks = [(o, t.size, r, io) for t, o, io in zip(texts, offs, iouts)]
    want = [O.bwt_aux(t, r)[1:] for t in texts]
    for plain in (True, False, False, False):
        dL.zero_(), dI.zero_(), dSA.zero_()
        assert eng.fwd(dT, dL, dI, blocks, dSA=dSA, plain=plain) == 0 and eng.wait()[0] == 0
        L, I, SA = dL.cpu().numpy(), dI.cpu().numpy(), dSA.cpu().numpy()
        for b, (t, o, io, (oU, oI)) in enumerate(zip(texts, offs, iouts, want)):
            assert np.array_equal(I[io:io + oI.size], oI), (plain, t.size)
            p0, col = int(oI[0]), L[o + b:o + b + t.size + 1]
            assert np.array_equal(np.concatenate([col[:p0], col[p0 + 1:]]), oU), (plain, t.size)
            sa = SA[o:o + t.size]
            assert np.array_equal(np.sort(sa), np.arange(t.size)), (plain, t.size)
    eng.close()
