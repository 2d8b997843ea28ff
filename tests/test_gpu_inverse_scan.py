"""The inverse's scan of chunk counts by one CTA or a cluster of CTAs per block (blocks averaging at most 64 chunks, or
more): batches on both sides of the line, with blocks of one chunk, of as many as a CTA has chunk groups, and of more."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [(1,), (64,), (65,), (1, 127), (1, 129), (257, 2, 1), (63, 64, 66), (129,) * 3])
def test_batches_around_the_line(chunks):
    import torch

    rng = np.random.default_rng(sum(chunks))
    offs, texts, off = [], [], 3
    for k, c in enumerate(chunks):  # 4096 bytes a chunk at these sizes; the last one ragged
        n = c * 4096 - (k * 1021 + 7) % 4094
        t = rng.integers(0, (256, 7)[k % 2], n).astype(np.uint8)
        t[n // 3:n // 2] = 200
        offs.append(off)
        texts.append(t)
        off += n + 1
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
