"""Inverse batches whose blocks are not listed by ascending offset: adjacent blocks in descending and shuffled order, one
that is no BWT among them, and a string listed twice. Each block's result is the one it has alone."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["descending", "shuffled", "bad", "twice"])
@pytest.mark.parametrize("sizes", [(100, 100), (2, 3, 5, 300, 4096, 2), (70_000, 4095, 130_001, 9, 33_000)])
def test_blocks_in_any_order(order, sizes):
    import torch

    rng = np.random.default_rng(sum(sizes))
    texts = [rng.integers(0, (256, 5)[k % 2], n).astype(np.uint8) for k, n in enumerate(sizes)]
    offs = np.concatenate([[0], np.cumsum(sizes)])[:-1] + 1  # adjacent, from an odd offset on
    U, want = np.zeros(sum(sizes) + 17, np.uint8), np.zeros(sum(sizes) + 17, np.uint8)
    blocks = []
    for t, o in zip(texts, offs):
        rc, u, i = O.bwt_aux(t, 1 << 30)
        assert rc == 0
        U[o:o + t.size], want[o:o + t.size] = u, t
        blocks.append((int(o), t.size, int(i[0])))
    bad = None
    if order == "bad":  # one byte value throughout has one psi cycle only with its primary index at n
        bad = int(np.argmax(sizes))
        o, n, _ = blocks[bad]
        U[o:o + n] = 7
        blocks[bad] = (o, n, n // 2 + 1)
        want[o:o + n] = 0
    blocks = blocks[::-1] if order == "descending" else [blocks[k] for k in rng.permutation(len(blocks))]
    if order == "twice":
        blocks = blocks + blocks[:2]
    dU = torch.from_numpy(U).cuda()
    eng = codec.Engine()
    for plain in (True, False, False, False):
        out = torch.zeros(U.size, dtype=torch.uint8, device="cuda")
        assert eng.inv(dU, out, blocks, plain=plain) == 0
        rc, status = eng.wait(len(blocks))
        got = out.cpu().numpy()
        if bad is None:
            assert rc == 0 and not status.any()
        else:
            assert rc == -1 and [int(s) for s in status] == [-1 if b[0] == offs[bad] else 0 for b in blocks]
            got[offs[bad]:offs[bad] + sizes[bad]] = 0
        assert np.array_equal(got, want)
    eng.close()
