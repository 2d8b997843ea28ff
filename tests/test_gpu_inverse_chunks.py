"""The inverse's psi build, chain walk, ranking and copy at the sizes where they change shape: chunk and tile edges
(4096 bytes, one tile per chunk on small batches), the steps of the mark density (128 KiB, 1.5 MiB, 4 MiB of input),
output blocks at every byte alignment, and strings with several cycles (not a BWT: reported, whatever the ranking meets
on them)."""
import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec

pytestmark = pytest.mark.gpu


def _text(n, seed):
    rng = np.random.default_rng(seed)
    t = rng.integers(0, (2, 5, 256)[seed % 3], n).astype(np.uint8)
    if n > 64:  # verbatim repeats: chains of equal bytes, long stretches between marks
        t[n // 2:n // 2 + n // 4] = t[:n // 4]
        t[-(n // 8):] = t[0]
    return t


@pytest.mark.parametrize("n", [2, 3, 5, 255, 4095, 4096, 4097, 8191, 65535, 65537, (128 << 10) - 1,
                               (128 << 10) + 1, (1 << 20) - 1, (1 << 20) + 1, (1536 << 10) + 1])
def test_round_trip_at_chunk_edges(n):
    T = _text(n, n)
    rc, U, I = O.bwt_aux(T, 1 << 30)
    assert rc == 0
    for _ in range(3):  # plain launches, then the captured graph
        rc, back = codec.unbwt_aux(U, n, I)
        assert rc == 0 and np.array_equal(back, T)


@pytest.mark.parametrize("total", [(4 << 20) - 3, (4 << 20) + 5])
def test_batch_around_a_mark_density_step(total):
    import torch

    sizes = [17, 4099, 70001, 300007, 3]
    sizes.append(total - sum(sizes))
    texts = [_text(n, 3 * k) for k, n in enumerate(sizes)]
    offs, off = [], 1
    for k, n in enumerate(sizes):  # every output alignment
        offs.append(off)
        off += n + 1 + k
    U, blocks = np.zeros(off + 16, np.uint8), []
    for t, o in zip(texts, offs):
        rc, u, i = O.bwt_aux(t, 1 << 30)
        assert rc == 0
        U[o:o + t.size] = u
        blocks.append((o, t.size, int(i[0])))
    dU = torch.from_numpy(U).cuda()
    out = torch.full((U.size,), 0xA5, dtype=torch.uint8, device="cuda")
    eng = codec.Engine()
    for plain in (True, False, False, False):
        out.fill_(0xA5)
        assert eng.inv(dU, out, blocks, plain=plain) == 0
        rc, status = eng.wait(len(blocks))
        assert rc == 0 and not status.any()
        got, want = out.cpu().numpy(), np.full(U.size, 0xA5, np.uint8)
        for t, o in zip(texts, offs):
            want[o:o + t.size] = t
        assert np.array_equal(got, want)  # nothing outside the blocks is touched
    eng.close()


@pytest.mark.parametrize("n", [64, 5000, 100_000, 1 << 20])
def test_several_cycles_are_reported(n):
    """A string sorted into one run per byte value: its rows fall into many short cycles."""
    U = np.sort(np.arange(n) % 251).astype(np.uint8)
    rc, back = codec.unbwt_aux(U, n, np.array([n // 2 + 1], np.int32))
    assert rc == -1
    T = _text(n, 1)  # the engine is fit for the next call
    rc, U, I = O.bwt_aux(T, 1 << 30)
    rc, back = codec.unbwt_aux(U, n, I)
    assert rc == 0 and np.array_equal(back, T)
