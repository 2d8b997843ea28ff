"""Results in host memory: blocks on both sides of the size from which the device writes the caller's pageable buffer
itself (512 KiB), fresh and touched pages, in place, page-locked, mixed in one batch; a rejected string leaves its buffer
alone; calls that follow each other without a wait, whose uploads share host tables; a stream under capture is refused
and the capture goes on."""
import ctypes

import numpy as np
import pytest

import oracle as O
from kolmo_gb300 import codec, native
from kolmo_gb300 import workloads as W

pytestmark = pytest.mark.gpu
EDGE = 512 << 10


def _call(name, src, dst, n, r, I):
    A = np.zeros(1, np.int32)
    return getattr(native.lib(), name)(src, dst, A.ctypes.data, n, r, I.ctypes.data, 1)


@pytest.mark.parametrize("where", ["fresh", "touched", "inplace", "locked"])
@pytest.mark.parametrize("n", [4096, EDGE - 1, EDGE, EDGE + 1, (1 << 20) + 7])
def test_single_calls(n, where):
    import torch

    T = W.logs(n, n)
    r = 1 << 16
    _, oU, oI = O.bwt_aux(T, r)
    for _ in range(3):
        lock = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        a = {"fresh": lambda: np.empty(n, np.uint8), "touched": lambda: np.full(n, 9, np.uint8),
             "inplace": lambda: T.copy(), "locked": lambda: lock.numpy()}[where]
        U, I = a(), np.zeros(oI.size, np.int32)
        src = U if where == "inplace" else T
        assert _call("kolmo_sais_bwt_aux", src.ctypes.data, U.ctypes.data, n, r, I) == 0
        assert np.array_equal(U, oU) and np.array_equal(I, oI)
        back = U.copy() if where == "inplace" else a()
        src = back if where == "inplace" else oU
        assert _call("kolmo_sais_unbwt_aux", src.ctypes.data, back.ctypes.data, n, r, I) == 0
        assert np.array_equal(back, T)


def test_batches_mix_staged_and_direct_blocks():
    sizes = [100, EDGE + 3, 17, 70_001, EDGE - 16, 2 * EDGE + 1, 16]
    texts = [W.source_block(k % 3, n, n) for k, n in enumerate(sizes)]
    want = [O.bwt_aux(t, 1 << 16) for t in texts]
    for pick in (range(len(sizes)), [0, 2, 3, 6], [1, 5]):
        rc, got = codec.fwd_batch([(texts[k], 1 << 16) for k in pick])
        assert rc == 0
        for k, (c, U, I) in zip(pick, got):
            assert c == 0 and np.array_equal(U, want[k][1]) and np.array_equal(I, want[k][2])
        rc, back = codec.inv_batch([(want[k][1], 1 << 16, want[k][2]) for k in pick])
        assert rc == 0
        for k, (c, t) in zip(pick, back):
            assert c == 0 and np.array_equal(t, texts[k])


@pytest.mark.parametrize("n", [5000, EDGE + 5])
def test_rejected_string_leaves_its_buffer(n):
    U = np.sort(np.arange(n) % 251).astype(np.uint8)
    out = np.full(n, 77, np.uint8)
    assert _call("kolmo_sais_unbwt_aux", U.ctypes.data, out.ctypes.data, n, n, np.array([n // 2 + 1], np.int32)) == -1
    assert (out == 77).all()


def test_calls_without_a_wait_between():
    import torch

    texts = [W.logs(40_000, 1), W.acgt(90_000, 2), W.logs(40_000, 3)]
    want = [O.bwt_aux(t, 1 << 12)[1:] for t in texts]
    eng, outs = codec.Engine(), []
    eng.fwd(torch.zeros(200_064, dtype=torch.uint8, device="cuda"), torch.zeros(200_001, dtype=torch.uint8, device="cuda"),
            torch.zeros(100, dtype=torch.int32, device="cuda"), [(0, 200_000, 1 << 12, 0)])
    for t in texts:  # different shapes: every upload has another table
        d = torch.zeros(t.size + 64, dtype=torch.uint8, device="cuda")
        d[:t.size] = torch.from_numpy(t).cuda()
        L = torch.zeros(t.size + 1, dtype=torch.uint8, device="cuda")
        I = torch.zeros(100, dtype=torch.int32, device="cuda")
        assert eng.fwd(d, L, I, [(0, t.size, 1 << 12, 0)]) == 0
        outs.append((d, L, I))
    assert eng.wait()[0] == 0
    inv = codec.Engine()
    keep = []
    for (d, L, I), t, (oU, oI) in zip(outs, texts, want):
        assert np.array_equal(I.cpu().numpy()[:oI.size], oI)
        u, o = torch.from_numpy(oU).cuda(), torch.zeros(t.size, dtype=torch.uint8, device="cuda")
        assert inv.inv(u, o, [(0, t.size, int(oI[0]))]) == 0
        keep.append((u, o))
    assert inv.wait(1)[0] == 0
    for (u, o), t in zip(keep, texts):
        assert np.array_equal(o.cpu().numpy(), t)


def test_capturing_stream_is_refused():
    import torch

    t = W.logs(30_000, 5)
    d = torch.zeros(t.size + 64, dtype=torch.uint8, device="cuda")
    d[:t.size] = torch.from_numpy(t).cuda()
    L = torch.zeros(t.size + 1, dtype=torch.uint8, device="cuda")
    I = torch.zeros(64, dtype=torch.int32, device="cuda")
    oU, oI = O.bwt_aux(t, 1 << 12)[1:]
    u, out = torch.from_numpy(oU).cuda(), torch.zeros(t.size, dtype=torch.uint8, device="cuda")
    eng, s, g = codec.Engine(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    fb, ib = [(0, t.size, 1 << 12, 0)], [(0, t.size, int(oI[0]))]
    assert eng.fwd(d, L, I, fb) == 0 and eng.wait()[0] == 0 and eng.inv(u, out, ib) == 0 and eng.wait(1)[0] == 0
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        L.zero_()
        rcs = eng.fwd(d, L, I, fb, stream=s), eng.inv(u, out, ib, stream=s)
    assert rcs == (-2, -2)
    g.replay()
    torch.cuda.synchronize()
    assert eng.fwd(d, L, I, fb) == 0 and eng.wait()[0] == 0
    assert np.array_equal(I.cpu().numpy()[:oI.size], oI)
