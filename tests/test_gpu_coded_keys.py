"""Round 0 on coded keys (KGBWT_OPT_LSD_BYTES = 8: the first 64 bits of the suffix in an order-preserving prefix code of
the block's bytes) against the oracle, exact, where the code or the key kernels can go wrong: alphabets of one, two, a
few and all byte values, weights that drive codewords to their longest, block lengths around the 16-position runs and
the 4096-suffix sort tiles, texts that end in their smallest byte (what the padding past the end reads as), and batches
whose blocks are packed, padded or start at odd offsets."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec
from kolmo_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = (2, 3, 15, 16, 17, 31, 33, 63, 64, 65, 255, 4095, 4096, 4097, 8191, 8193, 20011)


def _text(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "one":
        return np.full(n, 7, np.uint8)
    if kind == "two":  # 1-bit codewords: 64 bytes in a key
        return (rng.random(n) < 0.02).astype(np.uint8) * 255
    if kind == "skewed":  # every byte value; geometric weights drive codewords to the longest
        return np.minimum(rng.geometric(0.5, n) - 1, 255).astype(np.uint8) ^ (rng.random(n) < 0.02) * rng.integers(
            0, 256, n).astype(np.uint8)
    if kind == "uniform":
        return rng.integers(0, 256, n).astype(np.uint8)
    if kind == "tail":  # ends in its smallest byte, repeated as inside the text
        t = rng.integers(3, 6, n).astype(np.uint8)
        t[-min(n, 40):] = 3
        t[n // 3:n // 3 + min(n // 3, 200)] = 3
        return t
    if kind == "repeats":
        t = rng.integers(97, 101, max(n // 5, 1)).astype(np.uint8)
        return np.resize(t, n)
    return W.zipf_prose(n, seed, ncopies=3, copy_min=max(2, n // 50), copy_max=max(3, n // 9))


@pytest.mark.parametrize("kind", ["one", "two", "skewed", "uniform", "tail", "repeats", "prose"])
@pytest.mark.parametrize("gap", ["packed", "padded", "odd"])
def test_coded_round0_against_oracle(kind, gap):
    import torch

    texts = [np.ascontiguousarray(_text(kind, n, 100 + n)) for n in SIZES]
    off, offs = 8 if gap == "odd" else 0, []
    for k, t in enumerate(texts):
        offs.append(off)
        off += t.size if gap == "packed" else (t.size + 15) // 16 * 16 if gap == "padded" else t.size + 1 + k % 5
    buf = np.full(off + 64, 200, np.uint8)  # what lies between and past the blocks is not theirs
    for t, o in zip(texts, offs):
        buf[o:o + t.size] = t
    r, iouts, k = 1 << 6, [], 0
    for t in texts:
        iouts.append(k)
        k += (t.size - 1) // r + 1
    whole = torch.from_numpy(np.concatenate([np.zeros(8, np.uint8), buf])).cuda()
    dT = whole[8:]  # a text buffer that is 8-byte but not 16-byte aligned
    dL = torch.zeros(off + len(texts), dtype=torch.uint8, device="cuda")
    dI = torch.zeros(k, dtype=torch.int32, device="cuda")
    dSA = torch.zeros(off, dtype=torch.int32, device="cuda")
    eng = codec.Engine()
    eng.config(lsd_bytes=8)
    blocks = [(o, t.size, r, io) for t, o, io in zip(texts, offs, iouts)]
    for plain in (True, False, False, False):  # the graph is captured when the shape comes back
        for x in (dL, dI, dSA):
            x.zero_()
        assert eng.fwd(dT, dL, dI, blocks, dSA=dSA, plain=plain) == 0 and eng.wait()[0] == 0
        L, I, SA = dL.cpu().numpy(), dI.cpu().numpy(), dSA.cpu().numpy()
        for b, (t, o, io) in enumerate(zip(texts, offs, iouts)):
            oU, oI = O.bwt_aux(t, r)[1:]
            assert np.array_equal(I[io:io + oI.size], oI), (plain, t.size)
            p0, col = int(oI[0]), L[o + b:o + b + t.size + 1]
            assert np.array_equal(np.concatenate([col[:p0], col[p0 + 1:]]), oU), (plain, t.size)
            assert np.array_equal(np.sort(SA[o:o + t.size]), np.arange(t.size)), (plain, t.size)
    assert eng.last_config()["lsd_bytes"] == 8
    eng.close()
