"""Suffix arrays of the forward engine, entry by entry against the oracle's, on the texts that exercise round 0's coded keys
and the rank labels of large groups: a permutation with right U and samples can still order the members of a group
wrongly where their neighbours hold equal bytes."""
import numpy as np
import pytest

import oracle as O
import test_gpu_coded_keys as coded
import test_gpu_rank_labels as labels
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu

CASES = [(coded._text, k, (2, 17, 64, 255, 4097, 20011)) for k in ("one", "two", "skewed", "tail", "repeats", "prose")]
CASES += [(labels._text, k, (2049, 40_000, 100_003)) for k in ("period1", "period64", "period4097", "runs", "copies", "fibonacci")]


@pytest.mark.parametrize("text,kind,sizes", CASES, ids=[f"{t.__module__[9:]}-{k}" for t, k, _ in CASES])
@pytest.mark.parametrize("lsd_round0,lsd_bytes", [(1, 8), (1, 16), (0, 16)])
def test_suffix_array_is_exact(text, kind, sizes, lsd_round0, lsd_bytes):
    import torch

    texts = [np.ascontiguousarray(text(kind, n, 31 * n)) for n in sizes]
    # listed by descending offset, more bytes between them than there are blocks
    offs, off = [], 8
    for t in texts[::-1]:
        offs.insert(0, off)
        off += t.size + len(texts) + 3
    buf = np.full(off + 64, 99, np.uint8)
    for t, o in zip(texts, offs):
        buf[o:o + t.size] = t
    r = 1 << 20
    blocks = [(o, t.size, r, k) for k, (t, o) in enumerate(zip(texts, offs))]
    dT = torch.from_numpy(buf).cuda()
    dL = torch.zeros(off + 64, dtype=torch.uint8, device="cuda")
    dI = torch.zeros(len(texts), dtype=torch.int32, device="cuda")
    dSA = torch.zeros(off, dtype=torch.int32, device="cuda")
    want = [(O.suffix_array(t), *O.bwt_aux(t, r)[1:]) for t in texts]
    eng = codec.Engine()
    eng.config(lsd_round0=lsd_round0, lsd_bytes=lsd_bytes)
    for plain in (True, False, False):
        for x in (dL, dI, dSA):
            x.zero_()
        assert eng.fwd(dT, dL, dI, blocks, dSA=dSA, plain=plain) == 0 and eng.wait()[0] == 0
        L, I, SA = dL.cpu().numpy(), dI.cpu().numpy(), dSA.cpu().numpy()
        for b, (o, t, (sa, u, i)) in enumerate(zip(offs, texts, want)):
            assert np.array_equal(SA[o:o + t.size], sa), (plain, t.size)
            p0, col = int(i[0]), L[o + b:o + b + t.size + 1]
            assert I[b] == p0 and np.array_equal(np.concatenate([col[:p0], col[p0 + 1:]]), u), (plain, t.size)
    eng.close()
