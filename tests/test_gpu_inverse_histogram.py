"""The inverse's byte counts read 16-byte words between a block's unaligned ends: blocks of every alignment and of the
lengths around a word, a thread's words and a chunk, in one batch; and blocks of one long run."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(2, 3, 15, 16, 17, 31, 32, 33, 49), (4080, 4095, 4097, 8193, 16385)])
@pytest.mark.parametrize("values", [1, 3, 256])
def test_blocks_of_every_alignment(sizes, values):
    import torch

    rng = np.random.default_rng(len(sizes) * values)
    offs, texts, off = [], [], 0
    for n in sizes:
        for al in range(16):
            off += (al - off) % 16
            offs.append(off)
            texts.append(rng.integers(255 - values + 1, 256, n).astype(np.uint8))
            off += n
    U, blocks = np.zeros(off + 16, np.uint8), []
    for t, o in zip(texts, offs):
        rc, u, i = O.bwt_aux(t, 1 << 30)
        assert rc == 0
        U[o:o + t.size] = u
        blocks.append((o, t.size, int(i[0])))
    dU = torch.from_numpy(U).cuda()
    eng = codec.Engine()
    for plain in (True, False, False, False):
        out = torch.zeros(U.size, dtype=torch.uint8, device="cuda")
        assert eng.inv(dU, out, blocks, plain=plain) == 0
        rc, status = eng.wait(len(blocks))
        assert rc == 0 and not status.any()
        got, want = out.cpu().numpy(), np.zeros(U.size, np.uint8)
        for t, o in zip(texts, offs):
            want[o:o + t.size] = t
        assert np.array_equal(got, want)
    eng.close()
